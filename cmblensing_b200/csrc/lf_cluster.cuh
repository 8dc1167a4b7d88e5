// Cluster-resident LenseFlow: one whole RK4 integration per launch for N <= 256.
//
// A thread-block cluster of CL blocks integrates one component of one map
// from t0 to t1.  Block r owns rows [r RPC, (r+1) RPC) and packed columns
// [r KC, (r+1) KC) of the row spectra; the RK4 state (y0, acc) stays in
// registers, the row spectra in shared memory, and the two transpositions of
// a stage (rows -> columns before the column pass, back after it) are stores
// into the other blocks' shared memory, counted on the receiving block's
// mbarriers; a stage has no barrier of the cluster or of a block.
// Per stage HBM/L2 sees only the p planes.
//
// A group of TP = N / E lanes of one warp holds a length-N transform, E
// elements a lane (element lane + TP e in register e), and exchanges between
// radix passes through its own shared memory, so that the row and column
// phases need no block barrier at all.  Group g of a block owns row pair
// (2g, 2g + 1) in the row phase and column g in the column phase.
//
// Spectral conventions, the packed half spectra and the two right-hand sides
// are those of lf_kernels.cuh; as in its paired row passes every real
// transform is half of a complex one:
//   standard  Z = DX + i DY per row (inverse), w = y_a + i y_b per row pair
//   adjoint   Z = K_a + i K_b per row pair (inverse), w = (p_x + i p_y) y per row
#pragma once

#include "lf_kernels.cuh"

namespace lf {

// ------------------------------------------------------------ geometry
// Elements of a transform per lane: 16 (two radix passes, one exchange) where the registers allow it.
template <typename T, int N> __host__ __device__ constexpr int cl_elems() { return sizeof(T) == 4 && N >= 256 ? 16 : 8; }

template <typename T, int N, int CL> struct ClGeo {
  static constexpr int H = N / 2;
  static constexpr int E = cl_elems<T, N>();
  static constexpr int TP = N / E;       // lanes per transform
  static constexpr int G = N / (2 * CL);  // groups per block = row pairs = columns
  static constexpr int NT = G * TP;      // threads per block
  static constexpr int RPC = 2 * G;      // rows per block
  static constexpr int KC = G;           // packed columns per block
  static_assert(N == 64 || N == 128 || N == 256, "a group is at most one warp");
  static_assert(NT % 32 == 0 && CL > 1 && KC == 8, "whole warps, several blocks, 64-byte puts");
};

// Radices of the length-N group transform in forward order (the inverse runs them reversed): one pass of
// radix E, then r2 (then r3).
__host__ __device__ constexpr int cl_r2(int N, int E) { return E == 16 ? N / 16 : N == 128 ? 4 : 8; }
__host__ __device__ constexpr int cl_r3(int N, int E) { return N / (E * cl_r2(N, E)); }
// Pass table (W_{R NS}^{r k} at (r - 1) NS + k): forward (r2, E), (r3, E r2); inverse (r2, r3), (E, r2 r3).
// With two equal passes the inverse block is the forward one.
__host__ __device__ constexpr bool cl_shared_table(int N, int E) { return E * E == N; }
__host__ __device__ constexpr int cl_off_f3(int N, int E) { return (cl_r2(N, E) - 1) * E; }
__host__ __device__ constexpr int cl_off_i2(int N, int E) {
  return cl_shared_table(N, E) ? 0 : cl_off_f3(N, E) + (cl_r3(N, E) - 1) * E * cl_r2(N, E);
}
__host__ __device__ constexpr int cl_off_i3(int N, int E) {
  return cl_shared_table(N, E) ? 0 : cl_off_i2(N, E) + (cl_r2(N, E) - 1) * (cl_r3(N, E) > 1 ? cl_r3(N, E) : 0);
}
__host__ __device__ constexpr int cl_tw_size(int N, int E) {
  return N > 256 ? 0 : cl_shared_table(N, E) ? (E - 1) * E : cl_off_i3(N, E) + (E - 1) * (N / E);
}

// ------------------------------------------------------------- layouts
// Exchange scratch: element m of a transform sits at at(m) = sum over the set bits b of m of weight(b), a
// padded layout that is additive over disjoint bit fields, so that every access of a phase is one lane
// constant plus an immediate offset.  The weights (each larger than the sum of those before it) come from a
// search on a CPU model of the accesses: loads are free of bank conflicts, the exchange stores at most two
// ways (float32: 16 eight-byte slots per 128 bytes; float64: 8 sixteen-byte ones, none).  An XOR layout
// without any conflict spent an extra logic instruction on each access and the lane constants spilled.
template <typename T, int N> __host__ __device__ constexpr int lay_weight(int b) {
  constexpr int w32[3][8] = {{1, 2, 4, 12, 21, 42, 0, 0}, {1, 2, 4, 8, 18, 37, 76, 0}, {1, 2, 4, 8, 17, 34, 68, 136}};
  constexpr int w64[3][8] = {{1, 2, 4, 9, 18, 36, 0, 0}, {1, 2, 4, 9, 18, 36, 73, 0}, {1, 2, 4, 9, 18, 36, 72, 144}};
  constexpr int row = N == 64 ? 0 : N == 128 ? 1 : 2;
  return sizeof(T) == 4 ? w32[row][b] : w64[row][b];
}
// Elements of one transform's scratch, from row a's to row b's of a pair, and from one group's to the next.
// The step is at least the size and, modulo the slots, equal to the top bit's weight (see ColLay); two groups
// of eight lanes (float32, N = 64) share 128 bytes, so theirs start eight slots apart.
template <typename T, int N> __host__ __device__ constexpr int lay_size() {
  return sizeof(T) == 4 ? (N == 64 ? 83 : N == 128 ? 147 : 271) : (N == 64 ? 71 : N == 128 ? 144 : 287);
}
template <typename T, int N> __host__ __device__ constexpr int lay_step() {
  return sizeof(T) == 4 ? (N == 64 ? 90 : N == 128 ? 156 : 280) : (N == 64 ? 76 : N == 128 ? 145 : 288);
}
template <typename T, int N> __host__ __device__ constexpr int lay_group() {
  return sizeof(T) == 4 && N == 64 ? 184 : lay_step<T, N>() + lay_size<T, N>();
}
__host__ __device__ constexpr int log2_of(int n) { return n <= 1 ? 0 : 1 + log2_of(n / 2); }

// A row transform in one row's scratch.
template <typename T, int N> struct RowLay {
  static __host__ __device__ __forceinline__ constexpr int at(int m) {
    int x = 0;
#pragma unroll
    for (int b = 0; b < log2_of(N); ++b) x += ((m >> b) & 1) * lay_weight<T, N>(b);
    return x;
  }
};
// The column transform in the upper halves of a pair's two rows (the lower halves keep S or V): elements
// below N/2 in row a's, the others in row b's, one step further.
template <typename T, int N> struct ColLay {
  static __host__ __device__ __forceinline__ constexpr int at(int m) {
    int x = lay_weight<T, N>(log2_of(N) - 1) + ((m / (N / 2)) & 1) * lay_step<T, N>();
#pragma unroll
    for (int b = 0; b < log2_of(N) - 1; ++b) x += ((m >> b) & 1) * lay_weight<T, N>(b);
    return x;
  }
};
// Landing areas of the two transpositions: row spectra of all rows at this block's columns, [m][line], and Gx
// at this block's rows, [k][row].  What one block puts into a row of either area is one aligned run of 64
// bytes or more (a padded, unaligned layout took the transfers 1.3 times as long); an XOR of the line (row)
// with low bits of m (k) inside the run keeps a group's loads, consecutive m (k) at one line (row), free of
// bank conflicts.  Groups of sixteen lanes or more see those bits in the lane alone; with eight lanes
// (float32, N = 64) two groups share 128 bytes, one line (two rows) apart.
template <typename T, int N, int KC> __host__ __device__ __forceinline__ constexpr int col_at(int m, int line) {
  return m * KC + (line ^ (sizeof(T) == 8 ? m & 7 : N == 64 ? m & 6 : (m >> 1) & 7));
}
template <typename T, int N, int RPC> __host__ __device__ __forceinline__ constexpr int land_at(int k, int row) {
  return k * RPC + (row ^ (sizeof(T) == 8 ? k & 7 : N == 64 ? (k & 1) | ((k & 6) << 1) : k & 15));
}

// --------------------------------------------------- cluster primitives
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// the address in block ``rank`` of the cluster that corresponds to this block's shared address
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));  // (kept inside loops)
  return r;
}
// Hides a value's origin, so that what is derived from it is computed again in every iteration of a loop
// instead of being carried through it in registers (which then spill).
__device__ __forceinline__ void opaque(float& x) { asm volatile("" : "+f"(x)); }
__device__ __forceinline__ void opaque(double& x) { asm volatile("" : "+d"(x)); }
__device__ __forceinline__ void opaque(int& x) { asm volatile("" : "+r"(x)); }
// One complex value into another block's shared memory, counted as its bytes on that block's mbarrier.
__device__ __forceinline__ void cluster_put(uint32_t addr, uint32_t mbar, float2 v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(addr),
               "f"(v.x), "f"(v.y), "r"(mbar)
               : "memory");
}
__device__ __forceinline__ void cluster_put(uint32_t addr, uint32_t mbar, double2 v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(addr),
               "d"(v.x), "d"(v.y), "r"(mbar)
               : "memory");
}
// Wait for phase ``parity`` with cluster-scope acquire (the other blocks' puts), bounded like mbar_wait.
__device__ __forceinline__ bool cluster_mbar_wait(uint64_t* mbar, uint32_t parity, int tries) {
  const uint32_t addr = smem_addr(mbar);
  for (int i = 0; i < tries; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(addr), "r"(parity), "r"(1000u)
        : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The way out of a warp whose wait ran out.  The cluster's other warps miss its puts, so that their own next wait
// runs out too: each waits once more at most (about two seconds with its drain), puts nothing after that and comes
// here or has finished.  The barrier, which threads that have exited do not hold up, keeps every block's shared
// memory until the last put into it has been sent and drained.
__device__ __forceinline__ void cluster_leave() {  // (not .aligned: reached by a branch)
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// ------------------------------------------------------ group transforms
// One radix-R pass on registers: butterfly i of a lane is b = lane + TP i, its input r in register i + (E/R) r.
template <typename T, int N, int R, int NS, bool INV, int E>
__device__ __forceinline__ void cl_pass(c2<T> (&v)[E], const c2<T>* tw, int lane) {
  constexpr int TP = N / E, I = E / R;
#pragma unroll
  for (int i = 0; i < I; ++i) {
    c2<T> a[R];
#pragma unroll
    for (int r = 0; r < R; ++r) a[r] = v[i + I * r];
    if constexpr (NS > 1) {
      const int k = (lane + TP * i) % NS;
#pragma unroll
      for (int r = 1; r < R; ++r) a[r] = twmul<T, INV>(a[r], tw[(r - 1) * NS + k]);
    }
    dft<R, T, INV>(a);
#pragma unroll
    for (int r = 0; r < R; ++r) v[i + I * r] = a[r];
  }
}

// Between two passes: outputs of a radix-R pass after NS points to their natural positions, then back in
// lane order.  NV transforms at once, lay_step elements apart.  ``buf`` is the group's scratch.
template <typename T, int N, int R, int NS, class Lay, int NV, int E>
__device__ __forceinline__ void cl_exchange(c2<T> (&v)[NV][E], c2<T>* buf, int lane) {
  constexpr int TP = N / E, I = E / R, STEP = lay_step<T, N>();
  // positions are linear in the bits of the butterfly index b = lane + TP i: a lane part plus constants
  c2<T>* st = buf + Lay::at((lane / NS) * NS * R + lane % NS);
  const c2<T>* ld = buf + Lay::at(lane);
  __syncwarp();
#pragma unroll
  for (int q = 0; q < NV; ++q)
#pragma unroll
    for (int i = 0; i < I; ++i)
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int b = TP * i;
        st[Lay::at((b / NS) * NS * R + b % NS + r * NS) - Lay::at(0) + q * STEP] = v[q][i + I * r];
      }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < NV; ++q)
#pragma unroll
    for (int e = 0; e < E; ++e) v[q][e] = ld[Lay::at(TP * e) - Lay::at(0) + q * STEP];
}

// Unnormalised length-N transforms of NV register sets, natural order in and out (element lane + TP e in
// register e).
template <typename T, int N, class Lay, int NV, int E>
__device__ __forceinline__ void cl_fft(c2<T> (&v)[NV][E], c2<T>* buf, const c2<T>* tw, int lane) {
  constexpr int R2 = cl_r2(N, E), R3 = cl_r3(N, E);
#pragma unroll
  for (int q = 0; q < NV; ++q) cl_pass<T, N, E, 1, false>(v[q], tw, lane);
  cl_exchange<T, N, E, 1, Lay, NV>(v, buf, lane);
#pragma unroll
  for (int q = 0; q < NV; ++q) cl_pass<T, N, R2, E, false>(v[q], tw, lane);
  if constexpr (R3 > 1) {
    cl_exchange<T, N, R2, E, Lay, NV>(v, buf, lane);
#pragma unroll
    for (int q = 0; q < NV; ++q) cl_pass<T, N, R3, E * R2, false>(v[q], tw + cl_off_f3(N, E), lane);
  }
}

template <typename T, int N, class Lay, int NV, int E>
__device__ __forceinline__ void cl_ifft(c2<T> (&v)[NV][E], c2<T>* buf, const c2<T>* tw, int lane) {
  constexpr int R2 = cl_r2(N, E), R3 = cl_r3(N, E);
  if constexpr (R3 > 1) {
#pragma unroll
    for (int q = 0; q < NV; ++q) cl_pass<T, N, R3, 1, true>(v[q], tw, lane);
    cl_exchange<T, N, R3, 1, Lay, NV>(v, buf, lane);
#pragma unroll
    for (int q = 0; q < NV; ++q) cl_pass<T, N, R2, R3, true>(v[q], tw + cl_off_i2(N, E), lane);
    cl_exchange<T, N, R2, R3, Lay, NV>(v, buf, lane);
  } else {
#pragma unroll
    for (int q = 0; q < NV; ++q) cl_pass<T, N, R2, 1, true>(v[q], tw, lane);
    cl_exchange<T, N, R2, 1, Lay, NV>(v, buf, lane);
  }
#pragma unroll
  for (int q = 0; q < NV; ++q) cl_pass<T, N, E, N / E, true>(v[q], tw + cl_off_i3(N, E), lane);
}

template <typename T> __device__ __forceinline__ c2<T> shfl2(c2<T> v, int src, int width) {
  return mk<T>(__shfl_sync(0xffffffffu, v.x, src, width), __shfl_sync(0xffffffffu, v.y, src, width));
}

// ---------------------------------------------------- one system's pieces
// The shared memory and the phases of one integrated field (one component of one map).
//
// The two transpositions need no barrier: each value is put into its new owner's landing area and counted
// on the owner's mbarrier, and a block starts a phase when its area is complete.  That also orders the
// reuse of the areas: a block's Gx area is complete only after every block has read all of its columns, so
// the row phase may overwrite any column area, and a column area only after every block has read its Gx.
// (With a cluster barrier after each phase, membar and barrier stalls took a third of the time.)
template <typename T, int N, int CL> struct ClSystem {
  using G = ClGeo<T, N, CL>;
  using RL = RowLay<T, N>;
  using CO = ColLay<T, N>;
  static constexpr int E = G::E, HE = E / 2, TP = G::TP, H = G::H, RPC = G::RPC, KC = G::KC;
  static constexpr int STEP = lay_step<T, N>();
  static constexpr int kCol = N * KC, kLand = H * RPC, kRow = (G::G * lay_group<T, N>() + 1) & ~1;
  static constexpr int kElems = kCol + kLand + kRow;  // complex elements
  static constexpr uint32_t kPhaseBytes = uint32_t(N) * KC * sizeof(c2<T>);  // of either landing area

  c2<T>* row;   // this group's scratch; its rows' lower halves keep S (standard) or V (adjoint) between phases
  c2<T>* land;  // Gx of this block's rows
  c2<T>* col;   // row spectra of all rows, this block's columns
  uint64_t* mbar;  // [0] column area, [1] Gx area
  const c2<T>* tw;
  int g, lane;
  uint32_t rank;

  __device__ __forceinline__ void init(c2<T>* smem, uint64_t* bars, const c2<T>* table, int tid, uint32_t rk) {
    g = tid / TP;
    lane = tid % TP;
    col = smem;
    land = smem + kCol;
    row = smem + kCol + kLand + g * lay_group<T, N>();
    mbar = bars;
    tw = table;
    rank = rk;
  }

  // one thread, before the first cluster_sync
  __device__ __forceinline__ void init_barriers() const {
    for (int i = 0; i < 2; ++i) {
      mbar_init(mbar + i, 1);
      mbar_expect_tx(mbar + i, kPhaseBytes);
    }
  }
  // All of area ``which`` has landed for phase number ``phase``; ``more``: another phase follows.  False, for the
  // whole warp, if a lane's wait ran out: recorded, then drained like wait_or_record, and the warp leaves by
  // cluster_leave.
  __device__ __forceinline__ bool landed(int which, int phase, int polls, bool more) const {
    const bool ok = cluster_mbar_wait(mbar + which, phase & 1, polls);
    if (!ok) {
      record_timeout();
      cluster_mbar_wait(mbar + which, phase & 1, kWaitTries);
    }
    if (!__all_sync(0xffffffffu, ok)) return false;
    if (threadIdx.x == 0 && more) mbar_expect_tx(mbar + which, kPhaseBytes);
    return true;
  }
  __device__ __forceinline__ void put(c2<T>* local, uint32_t to, int which, c2<T> v) const {
    cluster_put(cluster_addr(smem_addr(local), to), cluster_addr(smem_addr(mbar + which), to), v);
  }

  // Column phase: Gx = IFFT(i KX / N^2 FFT(S)) of column g, to the blocks that own its rows.  ``before`` runs
  // ahead of the puts (global loads behind them would wait for the puts to drain).
  template <class Before> __device__ __forceinline__ void columns(T scale, Before before) const {
    c2<T> v[1][E];
#pragma unroll
    for (int e = 0; e < E; ++e) v[0][e] = col[col_at<T, N, KC>(lane, g) + TP * KC * e];
    cl_fft<T, N, CO, 1>(v, row, tw, lane);
    const int k = int(rank) * KC + g;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int m = lane + TP * e;
      const int kx = e < HE ? m : m - N;
      // zero on KX's Nyquist row of the packed DC/Nyquist column
      const T f = (e == HE && lane == 0 && k == 0) ? T(0) : scale * T(kx);
      v[0][e] = mk<T>(-f * v[0][e].y, f * v[0][e].x);
    }
    cl_ifft<T, N, CO, 1>(v, row, tw, lane);
    before();
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int m = lane + TP * e;
      put(land + land_at<T, N, RPC>(k, m % RPC), m / RPC, 1, v[0][e]);
    }
  }

  // The upper half (elements H..N-1) of a spectrum from the mirrored values q[e] = Z[N - k], k = lane + TP e,
  // e < E/2, that the lanes hold; ``nyq`` is Z[H] (lane 0).
  __device__ __forceinline__ void mirror(c2<T> (&v)[E], const c2<T> (&q)[HE], c2<T> nyq) const {
    const int src = (TP - lane) & (TP - 1);
#pragma unroll
    for (int e = HE; e < E; ++e) {
      const c2<T> x = shfl2<T>(q[E - 1 - e], src, TP);
      const c2<T> own = e == HE ? nyq : q[e == HE ? 0 : E - e];
      v[e] = lane == 0 ? own : x;
    }
  }

  // Standard right-hand side: v[q] = d_x y + i d_y y of rows 2g + q.
  __device__ __forceinline__ void inverse_std(c2<T> (&v)[2][E], T ky_scale) const {
    const c2<T>* kept = row + RL::at(lane);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      c2<T> up[HE], nyq = mk<T>(T(0), T(0));
#pragma unroll
      for (int e = 0; e < HE; ++e) {
        const int k = lane + TP * e;
        const c2<T> x = land[land_at<T, N, RPC>(lane, 2 * g + q) + RPC * TP * e];
        const c2<T> s = kept[RL::at(TP * e) + q * STEP];
        const T f = ky_scale * T(k);
        v[q][e] = mk<T>(x.x - f * s.x, x.y - f * s.y);        // DX + i DY, DY = i f S
        up[e] = mk<T>(x.x + f * s.x, -x.y - f * s.y);         // conj(DX) + i conj(DY)
        if (e == 0 && lane == 0) {  // packed real DC and Nyquist bins; the d_y spectrum has neither
          nyq = mk<T>(x.y, T(0));
          v[q][0] = mk<T>(x.x, T(0));
        }
      }
      mirror(v[q], up, nyq);
    }
    cl_ifft<T, N, RL, 2>(v, row, tw, lane);
  }

  // Adjoint right-hand side: v[0] = k_a + i k_b of rows 2g, 2g + 1, from K = Gx + i KY V / N.
  __device__ __forceinline__ void inverse_adj(c2<T> (&v)[1][E], T ky_scale) const {
    const c2<T>* kept = row + RL::at(lane);
    c2<T> up[HE], nyq = mk<T>(T(0), T(0));
#pragma unroll
    for (int e = 0; e < HE; ++e) {
      const int k = lane + TP * e;
      const T f = ky_scale * T(k);
      c2<T> kk[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const c2<T> x = land[land_at<T, N, RPC>(lane, 2 * g + q) + RPC * TP * e];
        const c2<T> s = kept[RL::at(TP * e) + q * STEP];
        kk[q] = (e == 0 && lane == 0) ? x : mk<T>(x.x - f * s.y, x.y + f * s.x);
      }
      v[0][e] = mk<T>(kk[0].x - kk[1].y, kk[0].y + kk[1].x);  // K_a + i K_b
      up[e] = mk<T>(kk[0].x + kk[1].y, kk[1].x - kk[0].y);    // conj(K_a) + i conj(K_b)
      if (e == 0 && lane == 0) {
        v[0][0] = mk<T>(kk[0].x, kk[1].x);
        nyq = mk<T>(kk[0].y, kk[1].y);
      }
    }
    mirror(v[0], up, nyq);
    cl_ifft<T, N, RL, 1>(v, row, tw, lane);
  }

  // Split the spectrum W of x + i y into the packed half spectra of x and y at k = lane + TP e, e < E/2.
  __device__ __forceinline__ void split(const c2<T> (&w)[E], c2<T> (&x)[HE], c2<T> (&y)[HE]) const {
    const int src = (TP - lane) & (TP - 1);
#pragma unroll
    for (int e = 0; e < HE; ++e) {
      c2<T> p = shfl2<T>(w[E - 1 - e], src, TP);
      if (lane == 0) p = e == 0 ? w[0] : w[(E - e) % E];
      const c2<T> b = cconj<T>(p);
      x[e] = cscale<T>(cadd<T>(w[e], b), T(0.5));
      const c2<T> d = csub<T>(w[e], b);
      y[e] = mk<T>(T(0.5) * d.y, T(-0.5) * d.x);  // (W - conj W') / 2i
      if (e == 0 && lane == 0) {
        x[0] = mk<T>(w[0].x, w[HE].x);
        y[0] = mk<T>(w[0].y, w[HE].y);
      }
    }
  }

  // Row spectrum values at k = lane + TP e of local row ``r`` to the owners of their columns.
  __device__ __forceinline__ void push(const c2<T> (&s)[HE], int r) const {
    const int m = int(rank) * RPC + r;
#pragma unroll
    for (int e = 0; e < HE; ++e) {
      const int k = lane + TP * e;
      put(col + col_at<T, N, KC>(m, k % KC), k / KC, 0, s[e]);
    }
  }

  // Standard: spectra of the next stage input's rows, w = y_a + i y_b: pushed, and kept at rest for d_y.
  __device__ __forceinline__ void forward_std(const T (&ya)[E], const T (&yb)[E]) const {
    c2<T> w[1][E], s[2][HE];
#pragma unroll
    for (int e = 0; e < E; ++e) w[0][e] = mk<T>(ya[e], yb[e]);
    cl_fft<T, N, RL, 1>(w, row, tw, lane);
    split(w[0], s[0], s[1]);
    push(s[0], 2 * g);
    push(s[1], 2 * g + 1);
    rest(s[0], s[1]);
  }

  // Adjoint: U = spectrum of p_x y (pushed) and V = spectrum of p_y y of rows 2g + q.  V replaces what the row's
  // scratch kept.
  __device__ __forceinline__ void forward_adj(const T (&y)[2][E], const T (&px)[2][E], const T (&py)[2][E]) const {
    c2<T> w[2][E], u[HE], vv[HE];
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int e = 0; e < E; ++e) w[q][e] = mk<T>(px[q][e] * y[q][e], py[q][e] * y[q][e]);
    cl_fft<T, N, RL, 2>(w, row, tw, lane);
    c2<T>* at = row + RL::at(lane);
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      split(w[q], u, vv);
      push(u, 2 * g + q);
#pragma unroll
      for (int e = 0; e < HE; ++e) at[RL::at(TP * e) + q * STEP] = vv[e];
    }
  }

  // The kept half spectra in the lower half of each row's scratch.  A lane reads back only what it wrote itself;
  // the barrier keeps the other lanes' last exchange reads ahead of the writes.
  __device__ __forceinline__ void rest(const c2<T> (&a)[HE], const c2<T> (&b)[HE]) const {
    c2<T>* at = row + RL::at(lane);
    __syncwarp();
#pragma unroll
    for (int e = 0; e < HE; ++e) {
      at[RL::at(TP * e)] = a[e];
      at[RL::at(TP * e) + STEP] = b[e];
    }
  }
};

// ------------------------------------------------------------ parameters
struct ClusterArgs {
  const void* f_in;  // [B][C][N][N] in the caller's dtype
  void* f_out;
  int in_f64, out_f64;
  const void* phi;  // derivative planes [B][5][N][N] of T
  const void* pp;   // p planes [B][2n+1][2][N][N] of T (PP), else null
  const void* tw;   // cl_tw_size(N, E) complex T
  double kbase;     // 2 pi / (N d)
  double t0, h;     // start time and signed step
  int nsteps, ncomp;
  int rev;          // time t0 + k h / 2 sits at p-plane index 2n - k instead of k
  void* ckpt;       // null, or y at the start of every step, [n][B C][N][N] of T
  void* save;       // SAVE (one step): of every stage, [4][B C] planes of T: d_x y, d_y y (standard) or y (adjoint)
  long planes;      // B C
};

// One RK4 stage update (util.py:184-199) of a pixel: rate k of stage s; returns the next stage input.
template <typename T> __device__ __forceinline__ T rk4_update(int s, T k, T h, T& y0, T& acc) {
  if (s < 3) {
    acc = s == 0 ? k : acc + T(2) * k;
    return y0 + (s == 2 ? h : T(0.5) * h) * k;
  }
  y0 = y0 + h / T(6) * (acc + k);
  return y0;
}

// ====================================================== the integration
// One cluster integrates component plane ``cmap`` over a.nsteps steps.  PP: p read from the p planes, else
// formed from the derivative planes when the stage time changes.  SAVE: the reverse passes' records of a
// single step, the standard system's stage gradients or the adjoint one's stage inputs.
template <typename T, int N, int CL, bool ADJ, bool PP, bool SAVE>
__device__ __forceinline__ void cl_integrate(const ClusterArgs& a, long cmap) {
  using G = ClGeo<T, N, CL>;
  using S = ClSystem<T, N, CL>;
  constexpr int E = G::E, TP = G::TP;
  constexpr int TW = cl_tw_size(N, E);
  constexpr long P = (long)N * N;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  c2<T>* data = reinterpret_cast<c2<T>*>(smem_raw);
  c2<T>* tw = data + S::kElems;
  uint64_t* mbar = reinterpret_cast<uint64_t*>(tw + TW);  // [0] the table, [1], [2] the landing areas
  static_assert(S::kElems * sizeof(c2<T>) % 16 == 0, "the table is copied to a 16-byte boundary");
  static_assert(TW * sizeof(c2<T>) % 16 == 0, "twiddle table: one bulk copy");
  const int tid = threadIdx.x;
  const uint32_t rank = cluster_rank();
  const long map = cmap / a.ncomp;
  S sys;
  sys.init(data, mbar + 1, tw, tid, rank);
  if (tid == 0) {
    mbar_init(mbar, 1);
    mbar_expect_tx(mbar, uint32_t(TW * sizeof(c2<T>)));
    bulk_g2s(tw, a.tw, TW * sizeof(c2<T>), mbar);
    sys.init_barriers();
  }
  const int polls = g_lf_wait_polls;
  const int lane = sys.lane;
  const long r0 = (long)rank * G::RPC + 2 * sys.g;  // first row of this group's pair
  const T ky_scale = T(a.kbase / double(N));
  const T kx_scale = T(a.kbase / (double(N) * double(N)));
  const T hh = T(a.h);
  const int K = 2 * a.nsteps;

  T px[2][E], py[2][E];
  auto load_p = [&](int k) {  // p at time t0 + k h / 2 of this lane's pixels
    if constexpr (PP) {
      const T* p = reinterpret_cast<const T*>(a.pp) + (map * (K + 1) + (a.rev ? K - k : k)) * 2 * P + r0 * N + lane;
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int e = 0; e < E; ++e) {
          px[q][e] = __ldg(p + q * N + TP * e);
          py[q][e] = __ldg(p + P + q * N + TP * e);
        }
    } else {
      const T* p = reinterpret_cast<const T*>(a.phi) + map * 5 * P + r0 * N + lane;
      const T t = T(a.t0 + k * (a.h * 0.5));
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const T* x = p + q * N + TP * e;
          p_vector<T>(__ldg(x), __ldg(x + P), __ldg(x + 2 * P), __ldg(x + 3 * P), __ldg(x + 4 * P), t, px[q][e],
                      py[q][e]);
        }
    }
  };

  T y0[2][E], acc[2][E];
  const long fo = cmap * P + r0 * N + lane;
  auto store = [&](T* plane, const T (&v)[2][E]) {  // this lane's pixels of a plane of the component
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int e = 0; e < E; ++e) plane[r0 * N + lane + q * N + TP * e] = v[q][e];
  };
  T* save = reinterpret_cast<T*>(a.save) + cmap * P * (ADJ ? 1 : 2);
  const long stage_planes = a.planes * P * (ADJ ? 1 : 2);
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const long i = fo + q * N + TP * e;
      y0[q][e] = a.in_f64 ? T(reinterpret_cast<const double*>(a.f_in)[i]) : T(reinterpret_cast<const float*>(a.f_in)[i]);
      acc[q][e] = T(0);
    }
  int k_now = -1;
  if constexpr (SAVE && ADJ) store(save, y0);
  cluster_sync();           // every block runs, with its barriers initialised, before anyone puts into it
  wait_or_record(mbar, 0);  // (a timed-out wait is recorded; the block goes on to its next wait)
  if constexpr (ADJ) {
    load_p(0);
    k_now = 0;
    sys.forward_adj(y0, px, py);
  } else {
    sys.forward_std(y0[0], y0[1]);
  }

#pragma unroll 1
  for (int it = 0; it < 4 * a.nsteps; ++it) {
    const int s = it & 3, i2 = 2 * (it >> 2);
    T kxs = kx_scale, kys = ky_scale;
    opaque(kxs);
    opaque(kys);
    const bool last = it == 4 * a.nsteps - 1;
    if constexpr (!ADJ && !SAVE) {
      if (s == 0 && a.ckpt) store(reinterpret_cast<T*>(a.ckpt) + ((it >> 2) * a.planes + cmap) * P, y0);
    }
    if (!sys.landed(0, it, polls, !last)) return cluster_leave();
    // p at the rate's time (standard) or at the next stage's (adjoint), needed when the columns have landed
    const int k = ADJ ? i2 + (s < 2 ? 1 : 2) : i2 + (s == 0 ? 0 : s < 3 ? 1 : 2);
    sys.columns(kxs, [&]() {
      if (k != k_now && !(ADJ && last)) {
        load_p(k);
        k_now = k;
      }
    });
    if (!sys.landed(1, it, polls, !last)) return cluster_leave();
    T yn[2][E];
    if constexpr (ADJ) {
      c2<T> v[1][E];
      sys.inverse_adj(v, kys);
#pragma unroll
      for (int e = 0; e < E; ++e) {
        yn[0][e] = rk4_update<T>(s, v[0][e].x, hh, y0[0][e], acc[0][e]);
        yn[1][e] = rk4_update<T>(s, v[0][e].y, hh, y0[1][e], acc[1][e]);
      }
      if (last) break;
      if constexpr (SAVE) store(save + (s + 1) * stage_planes, yn);
      sys.forward_adj(yn, px, py);
    } else {
      c2<T> v[2][E];
      sys.inverse_std(v, kys);
      if constexpr (SAVE) {
        T* gs = save + s * stage_planes + r0 * N + lane;
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
          for (int e = 0; e < E; ++e) {
            gs[q * N + TP * e] = v[q][e].x;
            gs[P + q * N + TP * e] = v[q][e].y;
          }
      }
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int e = 0; e < E; ++e)
          yn[q][e] = rk4_update<T>(s, px[q][e] * v[q][e].x + py[q][e] * v[q][e].y, hh, y0[q][e], acc[q][e]);
      if (last) break;
      sys.forward_std(yn[0], yn[1]);
    }
  }
  // (nothing is put into a block after its last Gx area has landed whole, so it may exit)
  if (!a.f_out) return;
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const long i = fo + q * N + TP * e;
      if (a.out_f64) reinterpret_cast<double*>(a.f_out)[i] = double(y0[q][e]);
      else reinterpret_cast<float*>(a.f_out)[i] = float(y0[q][e]);
    }
}

// The lens.  grid: one cluster per component of a map.
template <typename T, int N, int CL, bool ADJ, bool PP, int MINB>
__global__ void __launch_bounds__(ClGeo<T, N, CL>::NT, MINB) k_lens_cluster(ClusterArgs a) {
  cl_integrate<T, N, CL, ADJ, PP, false>(a, blockIdx.x / CL);
}

// n pixels of T to a caller's output of either type (an output that could not be written plane by plane).
template <typename T>
__global__ void __launch_bounds__(256) k_store_field(const T* src, void* dst, int dst_f64, long n) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    if (dst_f64) reinterpret_cast<double*>(dst)[i] = double(src[i]);
    else reinterpret_cast<float*>(dst)[i] = float(src[i]);
  }
}

// Measured, reference reverse pass of 16 TQU maps of 256^2, n = 7: row, column and accumulation launches per
// stage 3.35 ms; per step, with p formed from the derivative planes 3.1 ms, read from p planes 2.0 ms.
//
// One RK4 step of the two systems of a reverse pass, with the records that k_dphi_step needs: the field
// (standard) and the cotangent (adjoint), independent of one another within a step.  grid: two clusters per
// component of a map.  p from the step's p planes; float64 forms it itself (no room for them in its workspace).
template <typename T, int N, int CL, int MINB>
__global__ void __launch_bounds__(ClGeo<T, N, CL>::NT, MINB) k_vjp_step_cluster(ClusterArgs f, ClusterArgs d) {
  const long c = blockIdx.x / CL;
  constexpr bool PP = sizeof(T) == 4;
  if (c < f.planes) cl_integrate<T, N, CL, false, PP, true>(f, c);
  else cl_integrate<T, N, CL, true, PP, true>(d, c - f.planes);
}

// delta-phi accumulation of one RK4 step from the records of its four stages: the rate of k_dphi_accum
// (lense_flow.py:195-252) with the stage weights, summed in float64.  Adjoint stage j at time t + {0, 1/2,
// 1/2, 1} h pairs with standard stage j, or with 3 - j where that system ran the other way (``flip``).  One
// read and one write of the five accumulators per step instead of per stage, and the 2 x 2 inverse once per
// distinct time: bound by its bytes, 50 us a step for 16 TQU maps of 256^2 (256 MB, 5.1 TB/s) against 4 x 25 us
// by stages.  grads [4][B C][2][P], inputs [4][B C][P]; two pixels per thread.
// MINB 3 (80 registers, some spilled) where the grid fills the SMs several times over: reverse pass of 16 TQU maps
// of 256^2 1,980 -> 1,930 us, 32 T maps 1,880 -> 1,778, 64 QU maps of 128^2 1,288 -> 1,252; of 4 TQU maps of 256^2
// 569 -> 577, 2 of 128^2 206 -> 220.
template <typename T, int C, int MINB>
__global__ void __launch_bounds__(256, MINB) k_dphi_step(const T* __restrict__ grads, const T* __restrict__ inputs,
                                                   const T* __restrict__ phi, double* __restrict__ acc, int B, long P,
                                                   double t, double h, int flip, int first) {
  const long planes = (long)B * C, total = (long)B * P / 2;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const long b = 2 * i / P, px = 2 * i % P;
    const T* ph = phi + b * 5 * P + px;
    c2<T> g[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) g[j] = *reinterpret_cast<const c2<T>*>(ph + j * P);
    double sum[5][2] = {};
#pragma unroll
    for (int k = 0; k < 3; ++k) {  // the distinct times: adjoint stages {0}, {1, 2}, {3}
      double f[2][2] = {};         // fdf = sum of weight x delta x gradient, (x, y) of the two pixels
#pragma unroll
      for (int j = k == 0 ? 0 : 2 * k - 1; j <= (k == 0 ? 0 : k == 1 ? 2 : 3); ++j) {
        const double w = k == 1 ? 2.0 : 1.0;
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const long pl = b * C + c;
          const c2<T> d = *reinterpret_cast<const c2<T>*>(inputs + (j * planes + pl) * P + px);
          const T* gp = grads + ((flip ? 3 - j : j) * planes + pl) * 2 * P + px;
          const c2<T> gx = *reinterpret_cast<const c2<T>*>(gp), gy = *reinterpret_cast<const c2<T>*>(gp + P);
          f[0][0] += w * double(d.x) * double(gx.x);
          f[0][1] += w * double(d.x) * double(gy.x);
          f[1][0] += w * double(d.y) * double(gx.y);
          f[1][1] += w * double(d.y) * double(gy.y);
        }
      }
      const double tt = t + 0.5 * k * h;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const double gx = q ? g[0].y : g[0].x, gy = q ? g[1].y : g[1].x, gxx = q ? g[2].y : g[2].x,
                     gxy = q ? g[3].y : g[3].x, gyy = q ? g[4].y : g[4].x;
        const double mxx = 1.0 + tt * gxx, mxy = tt * gxy, myy = 1.0 + tt * gyy;
        const double inv = 1.0 / (mxx * myy - mxy * mxy + 1e-12);
        const double ixx = myy * inv, ixy = -mxy * inv, iyy = mxx * inv;
        const double ax = ixx * f[q][0] + ixy * f[q][1], ay = ixy * f[q][0] + iyy * f[q][1];
        const double pxv = gx * ixx + gy * ixy, pyv = gx * ixy + gy * iyy;
        sum[0][q] += ax;
        sum[1][q] += ay;
        sum[2][q] += tt * pxv * ax;
        sum[3][q] += tt * (pxv * ay + pyv * ax);
        sum[4][q] += tt * pyv * ay;
      }
    }
    const double w6 = h / 6.0;
    double* o = acc + b * 5 * P + px;
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      double2* oj = reinterpret_cast<double2*>(o + j * P);
      const double2 old = first ? make_double2(0.0, 0.0) : *oj;
      *oj = make_double2(old.x + w6 * sum[j][0], old.y + w6 * sum[j][1]);
    }
  }
}

}  // namespace lf
