// The two tile passes of a fused pseudo-spectral step on an N^3 grid, N = 32 YB.
//
// The 3D transform is split so that no tile needs data of another block: y =
// YB j1 + j2 and ky = k1 + 32 k2 (0 <= j1, k1 < 32, 0 <= j2, k2 < YB), and
//
//   plane passes  : one tile = the 32 rows y = YB j1 + j2 (j2 fixed) of an
//                   x-plane. In shared memory: the z transform of the rows
//                   (R2C / C2R) and the 32-point part of the y transform
//                   (j1 <-> k1), with a pointwise prologue or epilogue on the
//                   real values.
//   pencil passes : one tile = C spectral columns of one k1, all x and all j2:
//                   the YB-point rest of the y transform (j2 <-> k2), the
//                   x transform, a per-spectral-point operator (gradient step,
//                   G multiply, preconditioner, SPM force update, ...) with
//                   reductions, and back.
//
// Between them the data lies in a scratch array in pencil-tile order,
// [k1][column / C][j2][x][column % C] (scratch_index): a pencil tile is
// contiguous, a plane tile is 32-byte (or longer) runs. Every pass writes a
// tile to the addresses it read it from, so one scratch array per field
// serves a whole chain and half as much data competes for L2. All passes are
// persistent grids of independent blocks (no clusters): with the whole
// y transform in one pass a tile was an x-plane spread over the CTAs of a
// cluster, and their two exchanges (through distributed shared memory or L2)
// took most of the pass: 184 us at 256^3 FP64 for the inverse -> forward pass.
//
// Every kernel first checks the optional "go" word so that a chain of steps
// enqueued ahead stops exactly where the reference's loop would (LPsrc.cpp:52).
#pragma once

#include "fft_core.cuh"

namespace spm {

template <int N> struct Geo {
  static_assert(N % 32 == 0 && N >= 32 && N <= 256, "grid size must be a multiple of 32 in [32, 256]");
  static constexpr int M = N / 2;    // complex points per packed z-line
  static constexpr int YB = N / 32;  // points of the y transform's second part
  static constexpr int N1 = M / 8;   // z = 8 x N1
  static constexpr int M1 = N / 16;  // x = 16 x M1
};

// ------------------------------------------------------------------ geometry
// Spectral columns per pencil tile: 32 bytes. (Tiles of four FP64 columns, half
// as many blocks per SM: 115 -> 129 us a gradient step at 192^3, equal at 128^3
// and 160^3; at 256^3 one block of 512 threads per SM instead of two of 256.)
template <class T> constexpr int tile_cols() { return (int)(32 / sizeof(c2<T>)); }

// Position of (k1, column, j2, x) in the scratch array.
template <int N, int R = kRun>
__device__ __forceinline__ size_t scratch_index(int k1, int col, int j2, int x) {
  constexpr int M = Geo<N>::M, YB = Geo<N>::YB;
  return (((size_t)(k1 * (M / R) + col / R) * YB + j2) * N + x) * R + col % R;
}

// Position of the state value (kx, ky = k1 + 32 k2, column): in a packed
// spectrum, or in tile order, where a pencil tile's state is contiguous.
template <int N, class T> __device__ __forceinline__ size_t state_index(int k1, int k2, int kx, int col, int tiled) {
  return tiled ? scratch_index<N, tile_cols<T>()>(k1, col, k2, kx) : ((size_t)kx * N + k1 + 32 * k2) * Geo<N>::M + col;
}
template <int N, class T> __device__ __forceinline__ size_t state_kx_stride(int tiled) {
  return tiled ? (size_t)tile_cols<T>() : (size_t)N * Geo<N>::M;
}

// Groups per block of the plane passes that read the scratch (plane_inv,
// plane_inv_fwd) at 256^3 FP64: a block of 512 threads (one per SM) is two
// groups of N threads that work on tiles of their own with barriers of their
// own, and share one 64 KB stage in shared memory into which the next tile is
// copied (one tensor copy) while the groups compute. Two blocks of one group each
// with loads into registers (every tile waits for its loads): 113 against
// 101 us for the joint pass. Smaller grids run as fast without (their
// scratch stays in L2), and so does plane_fwd (contiguous rows); the pencil pass
// was slower staged (141 against 132 us: 32-byte rows, and the stage leaves
// the L1 too small for the state's loads).
template <int N, class T> constexpr int inv_groups() { return sizeof(T) == 8 && N == 256 ? 2 : 1; }

// The states of a pencil pass carry an L2 evict-first policy where the scratch
// fits in the 126 MB L2 but not beside a state of its size (FP64: 192^3, 2 x 57
// MB): the scratch then stays. Measured (gradient step, without and with): 192^3
// 108 and 104 us; 256^3, whose scratch does not fit by itself, 225 and 239 us. In
// FP32 (force steps only) the rule holds at 256^3: ten spring-pair iterations
// 13.80 and 13.77 ms.
template <int N, class T> constexpr bool stream_state() {
  constexpr size_t S = sizeof(T) * (size_t)N * N * N;
  return S < ((size_t)100 << 20) && 2 * S > ((size_t)100 << 20);
}

// Plane pass: N threads per tile of 32 rows x M complex values (16 per
// thread), rows padded by one value. 512 threads per SM in FP64 (up to 128
// registers each), 1024 in FP32. G: groups per block (inv_groups).
template <int N, class T, int GR = 1> struct PlaneGeo {
  static constexpr int TH = N, G = GR;
  static constexpr int STAGE = G > 1 ? kRows * Geo<N>::M : 0;
  static constexpr int RS = Geo<N>::M + 1;  // row stride
  static constexpr int UNITS = kRows * RS;
  static constexpr int TILES = N * Geo<N>::YB;  // per field
  static constexpr int CPS = (sizeof(T) == 8 ? 512 : 1024) / (G * N);
};
template <int N, class T, int G = 1> constexpr size_t plane_smem() {
  using PG = PlaneGeo<N, T, G>;
  return sizeof(c2<T>) * (N + PG::STAGE + G * PG::UNITS) + G * sizeof(double) * 32 * kRedMax + (G > 1 ? 16 * G + 128 : 0);
}

// Pencil pass: 16 YB C threads per tile of N x YB x C complex values; the
// exchange buffer pads each run of M1 C values by C.
template <int N, class T> struct PencilGeo {
  static constexpr int C = tile_cols<T>();
  static constexpr int YB = Geo<N>::YB;
  static constexpr int TH = 16 * YB * C;
  static constexpr int KS = (Geo<N>::M1 + 1) * C;  // stride of k1x
  static constexpr int JS = 16 * KS;               // stride of j2 / k2
  static constexpr int UNITS = YB * JS;
  static constexpr int NCG = Geo<N>::M / C;        // column groups
  static constexpr int TILES = 32 * NCG;           // per field
  static constexpr int CPS0 = (sizeof(T) == 8 ? 512 : 1024) / TH;
  static constexpr int CPS = CPS0 < 1 ? 1 : (CPS0 > 16 ? 16 : CPS0);
};
template <int N, class T> constexpr size_t pencil_smem() {
  return sizeof(c2<T>) * (N + PencilGeo<N, T>::UNITS) + sizeof(double2) * (N / 2 + 1) +
         sizeof(double) * 32 * kRedMax;
}

// The stage shared by a block's G groups: group g has a "full" barrier
// (completed by the copy's bytes) and an "empty" one (an arrival per warp of the
// group that has read its tile). The copy of the block's tile i + 1 is issued
// by the group of tile i once that group has read its own. Once a wait has given
// up (*err) no copy is issued any more.
template <int N, int G> struct Stage {
  uint64_t *full, *empty;  // [G]
  int *err;
  volatile int *issued;  // [G] copies issued into `full`; each count has one writer at a time
  __device__ void init(uint64_t *bars, int *s_ctl) {
    full = bars;
    empty = bars + G;
    err = s_ctl;
    issued = s_ctl + 1;
    if (threadIdx.x == 0) {
      for (int g = 0; g < G; g++) {
        mbar_init(full + g, 1);
        mbar_init(empty + g, N / 32);
        issued[g] = 0;
      }
      *err = 0;
      fence_barrier_init();
    }
  }
  // The group's tile of round `round` has arrived.
  __device__ void wait(int g, int round) { mbar_wait(full + g, round & 1, err); }
  // This warp has read it; thread 0 of the group then issues the next copy.
  template <class F> __device__ void next(int g, int tid, int round, F issue) {
    __syncwarp();
    if ((tid & 31) == 0) mbar_arrive(empty + g);
    if (tid == 0 && mbar_wait(empty + g, round & 1, err)) {
      fence_proxy_async();
      issue((g + 1) % G);
    }
  }
  // At the end, by one thread, once no group issues any more.
  __device__ void drain() const {
    for (int g = 0; g < G; g++) drain_copies(full + g, issued[g]);
  }
};

// The fields of a launch share its grid field-fastest: the blocks that work on
// the same tiles of the fields of a block run together, so that what the fields
// share (phi of Hessian products, the tangent of force steps) is read from
// memory once. Which tiles a block takes does not depend on the number of fields.
__device__ __forceinline__ int field_id() { return blockIdx.x; }
__device__ __forceinline__ int block_id() { return blockIdx.y; }
__device__ __forceinline__ int block_count() { return gridDim.y; }

// --------------------------------------------------------------- plane phases
// One tile in three phases per direction, each on registers with one exchange
// through `buf` in between (row r = j1, RS values apart):
//   y phase     : thread (q, b) holds 16 values of spectral column q. The
//                 32-point transform is 16 x 2: thread b transforms the rows
//                 2a + b, and the two threads of a column (lanes 16 apart)
//                 swap half of their values by shuffles for the radix 2.
//   class phase : thread (r, w), lane = row r, warp w: the z points q = a and
//                 q = N1 - a (mod N1), a = w (warp 0: the classes 0 and N1/2).
//                 Both members of every pair (q, M - q) are in the thread, so
//                 the R2C / C2R combinations need no exchange, and the
//                 twiddles are the same for a whole warp. 8-point transforms.
//   row phase   : task (r, jz): z points j = 8 j1z + jz, N1-point transforms,
//                 and the pointwise work on the real pairs (2j, 2j + 1).
// A value's slot in its row is 8 (q mod N1) + (q / N1) rotated by q mod N1: a
// class-phase thread reads and writes the same slots, a row-phase task too, so
// those phases need no barrier inside, and every phase reads and writes
// without bank conflicts at N = 128 and 256 (two-way in some phases elsewhere).
template <int N, class T> struct Plane {
  using G = Geo<N>;
  using T2 = c2<T>;
  static constexpr int M = G::M, N1 = G::N1, YB = G::YB;
  static constexpr int TH = PlaneGeo<N, T>::TH, RS = PlaneGeo<N, T>::RS;
  static constexpr int TASKS = kRows * 8;                 // row-phase tasks
  static constexpr int TPT = (TASKS + TH - 1) / TH;       // per thread

  __device__ static int slot(int a, int k2) { return a * 8 + ((k2 + a) & 7); }

  // y -> scratch: buf holds (row j1, q); writes the k1 values of column q.
  __device__ static void y_fwd(const T2 *buf, const T2 *tw, int tid, T2 *dst, int x, int j2) {
    const int b = (tid >> 4) & 1, q = (tid >> 5) * 16 + (tid & 15);
    const T2 *col = buf + b * RS + slot(q % N1, q / N1);
    T2 v[16];
#pragma unroll
    for (int a = 0; a < 16; a++) v[a] = col[2 * a * RS];
    // thread b = 1 keeps the upper half of the transform: with the odd inputs
    // negated, output i is that of i + 8 (mod 16)
#pragma unroll
    for (int a = 1; a < 16; a += 2) v[a] = flip_if(v[a], b);
    Dft<-1, 16, T2>::run(v);
    T2 *o = dst + scratch_index<N>(8 * b, q, j2, x);
    constexpr size_t KST = (size_t)M * YB * N;  // stride of k1
#pragma unroll
    for (int i = 0; i < 8; i++) {  // k1 = 8 b + i and 8 b + i + 16
      const T2 r = shfl_xor(v[8 + i], 16);
      const T2 u0 = b ? r : v[i];
      const T2 u1 = cmul(b ? v[i] : r, tw[(8 * b + i) * YB]);
      o[i * KST] = cadd(u0, u1);
      o[(i + 16) * KST] = csub(u0, u1);
    }
  }

  // scratch -> y: the inverse of y_fwd (unnormalised). o: the values k1 = 8 b,
  // 8 b + 1, ... of column q, kst apart (in the scratch or the stage); read()
  // is called when they have been loaded.
  template <class F> __device__ static void y_inv(T2 *buf, const T2 *tw, int tid, const T2 *o, size_t kst, F read) {
    const int b = (tid >> 4) & 1, q = (tid >> 5) * 16 + (tid & 15);
    T2 lo[8], v[16];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      lo[i] = o[i * kst];
      v[i] = o[(i + 16) * kst];
    }
    read();
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const T2 s = cadd(lo[i], v[i]);
      const T2 d = cmulc(csub(lo[i], v[i]), tw[(8 * b + i) * YB]);
      v[i] = b ? d : s;
      v[8 + i] = shfl_xor(b ? s : d, 16);
    }
    // thread b = 1 holds its inputs rotated by 8: the odd outputs change sign
    Dft<+1, 16, T2>::run(v);
    T2 *col = buf + b * RS + slot(q % N1, q / N1);
#pragma unroll
    for (int a = 0; a < 16; a++) col[2 * a * RS] = (a & 1) ? flip_if(v[a], b) : v[a];
  }

  // Forward class phase: twiddles, 8-point transforms, and the R2C combination
  //   2 X_q = (Z_q + conj Z_{M-q}) - i w^q (Z_q - conj Z_{M-q}), w = exp(-2 pi i / N)
  // (the values keep the factor 2; KParams::fscale takes it out).
  // X_{M-q} is conj of the same terms with the other sign.
  __device__ static void class_fwd(T2 *buf, const T2 *tw, int tid) {
    const int w = tid >> 5;
    T2 *row = buf + (tid & 31) * RS;
    const int a0 = w, a1 = w ? N1 - w : N1 / 2;
    T2 u[8], v[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      u[j] = row[slot(a0, j)];
      v[j] = row[slot(a1, j)];
    }
    if (w)
#pragma unroll
      for (int j = 1; j < 8; j++) u[j] = cmul(u[j], tw[2 * a0 * j]);
#pragma unroll
    for (int j = 1; j < 8; j++) v[j] = cmul(v[j], tw[2 * a1 * j]);
    Dft<-1, 8, T2>::run(u);
    Dft<-1, 8, T2>::run(v);
    if (w) {
#pragma unroll
      for (int k = 0; k < 8; k++) r2c_pair(u[k], v[7 - k], tw[a0 + N1 * k]);
    } else {
      u[0] = T2{(T)2 * (u[0].x + u[0].y), (T)2 * (u[0].x - u[0].y)};  // 2 (X_0 + i X_{N/2}), both real
#pragma unroll
      for (int k = 1; k < 4; k++) r2c_pair(u[k], u[8 - k], tw[N1 * k]);
      u[4] = T2{(T)2 * u[4].x, -(T)2 * u[4].y};
#pragma unroll
      for (int k = 0; k < 4; k++) r2c_pair(v[k], v[7 - k], tw[N1 / 2 + N1 * k]);
    }
#pragma unroll
    for (int k = 0; k < 8; k++) {
      row[slot(a0, k)] = u[k];
      row[slot(a1, k)] = v[k];
    }
  }
  // (Z_q, Z_{M-q}) -> 2 (X_q, X_{M-q}), w = w^q
  __device__ static void r2c_pair(T2 &p, T2 &m, T2 w) {
    const T2 e = {p.x + m.x, p.y - m.y};
    const T2 o = cmul(T2{p.y + m.y, m.x - p.x}, w);
    p = cadd(e, o);
    m = T2{e.x - o.x, o.y - e.y};
  }
  // (X_q, X_{M-q}) -> (Z_q, Z_{M-q}): Z_q = (X_q + conj X_{M-q}) + i w^{-q} (X_q - conj X_{M-q})
  __device__ static void c2r_pair(T2 &p, T2 &m, T2 w) {
    const T2 e = {p.x + m.x, p.y - m.y};
    const T2 o = cmulc(T2{p.x - m.x, p.y + m.y}, w);
    p = T2{e.x - o.y, e.y + o.x};
    m = T2{e.x + o.y, o.x - e.y};
  }

  // Inverse class phase: C2R combination, 8-point transforms, twiddles.
  __device__ static void class_inv(T2 *buf, const T2 *tw, int tid) {
    const int w = tid >> 5;
    T2 *row = buf + (tid & 31) * RS;
    const int a0 = w, a1 = w ? N1 - w : N1 / 2;
    T2 u[8], v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      u[k] = row[slot(a0, k)];
      v[k] = row[slot(a1, k)];
    }
    if (w) {
#pragma unroll
      for (int k = 0; k < 8; k++) c2r_pair(u[k], v[7 - k], tw[a0 + N1 * k]);
    } else {
      u[0] = T2{u[0].x + u[0].y, u[0].x - u[0].y};  // from X_0 + i X_{N/2}
#pragma unroll
      for (int k = 1; k < 4; k++) c2r_pair(u[k], u[8 - k], tw[N1 * k]);
      u[4] = T2{(T)2 * u[4].x, -(T)2 * u[4].y};
#pragma unroll
      for (int k = 0; k < 4; k++) c2r_pair(v[k], v[7 - k], tw[N1 / 2 + N1 * k]);
    }
    Dft<+1, 8, T2>::run(u);
    Dft<+1, 8, T2>::run(v);
    if (w)
#pragma unroll
      for (int j = 1; j < 8; j++) u[j] = cmulc(u[j], tw[2 * a0 * j]);
#pragma unroll
    for (int j = 1; j < 8; j++) v[j] = cmulc(v[j], tw[2 * a1 * j]);
#pragma unroll
    for (int j = 0; j < 8; j++) {
      row[slot(a0, j)] = u[j];
      row[slot(a1, j)] = v[j];
    }
  }

  // Row phase: body(e, r, jz, load, store) runs for each of the thread's tasks.
  template <class F> __device__ static void rows(int tid, F body) {
#pragma unroll
    for (int t = 0; t < TPT; t++) {
      const int e = tid + TH * t;
      if (TASKS % TH == 0 || e < TASKS) body(e >> 3, e & 7);
    }
  }
  __device__ static void row_load_inv(const T2 *buf, int r, int jz, T2 (&v)[N1]) {
    sfor<0, N1>([&](auto A) { v[SPM_CI(A)] = buf[r * RS + slot(SPM_CI(A), jz)]; });
    Dft<+1, N1, T2>::run(v);  // v[j1z]: complex z point 8 j1z + jz
  }
  __device__ static void row_store_fwd(T2 *buf, int r, int jz, T2 (&v)[N1]) {
    Dft<-1, N1, T2>::run(v);
    sfor<0, N1>([&](auto A) { buf[r * RS + slot(SPM_CI(A), jz)] = v[SPM_CI(A)]; });
  }
};

// Field arrays a policy reads beside its input (p.aux0, p.aux1): X::AUX, else none.
template <class X, class = void> struct AuxOf : std::integral_constant<int, 0> {};
template <class X> struct AuxOf<X, std::void_t<decltype(X::AUX)>> : std::integral_constant<int, X::AUX> {};

// The slot of the scalar block that an operator needs from the launch before: X::PRE,
// else none (-1).
template <class X, class = void> struct PreOf : std::integral_constant<int, -1> {};
template <class X> struct PreOf<X, std::void_t<decltype(X::PRE)>> : std::integral_constant<int, X::PRE> {};

// Asks for the 32 rows of tile (x, j2) of a real field to be brought into L2 (one
// warp; bulk prefetches want 16-byte alignment, which FP32 fields need not have).
// From 96^3 to 192^3 only (Hessian products in blocks of 8, FP64, without and
// with: 96^3 19.8 / 19.0, 128^3 38 / 35, 160^3 78 / 75, 192^3 151 / 136 us each;
// but 64^3 6.8 / 7.2 and 256^3 278 / 281 us, one product 320 / 335).
template <int N, class T> __device__ __forceinline__ void prefetch_rows(const void *field, int tid, int x, int j2) {
  if (N >= 96 && N <= 192 && ((uintptr_t)field & 15u) == 0 && field && tid < kRows)
    prefetch_l2(reinterpret_cast<const T *>(field) + ((size_t)x * N + Geo<N>::YB * tid + j2) * N, N * sizeof(T));
}

// A plane kernel's loop over the tiles of this thread's group: tiles vb + i G
// block_count(), vb = block_id() + g block_count() (what a grid of G block_count() one-group
// blocks does, so that the sums are the same). With INV the tile's input comes
// through the stage (or straight from the scratch, G = 1), and body(x, j2)
// follows the inverse class phase.
template <int N, class T, bool INV, int G> struct PlaneLoop {
  using T2 = c2<T>;
  using PG = PlaneGeo<N, T, G>;
  using P = Plane<N, T>;
  T2 *tw, *buf, *stage;
  double *red;
  int g, tid;
  Stage<N, G> st;
  __device__ PlaneLoop(unsigned char *raw, int *s_ctl) {
    stage = reinterpret_cast<T2 *>(G > 1 ? smem_base128(raw) : raw);
    tw = stage + PG::STAGE;
    T2 *work = tw + N;
    double *reds = reinterpret_cast<double *>(work + G * PG::UNITS);
    g = G > 1 ? threadIdx.x / N : 0;
    tid = G > 1 ? threadIdx.x % N : threadIdx.x;
    buf = work + g * PG::UNITS;
    red = reds + g * 32 * kRedMax;
    if constexpr (G > 1) st.init(reinterpret_cast<uint64_t *>(reds + G * 32 * kRedMax), s_ctl);
  }
  // barrier of the threads that share a tile
  __device__ void sync() const {
    if constexpr (G > 1) bar_sync(1 + g, N);
    else __syncthreads();
  }
  template <int AUX = 0, class F> __device__ void run(const TileParams<G> &p, int b, F body) {
    const T2 *src = reinterpret_cast<const T2 *>(p.in[b]);
    auto issue = [&](int tile, int gg) {
      if constexpr (G > 1) {
        if (tile >= PG::TILES) return;
        st.issued[gg] = st.issued[gg] + 1;
        mbar_expect_tx(st.full + gg, (unsigned)(PG::STAGE * sizeof(T2)));
        tma_load_4d(stage, &p.tm[b], 0, (tile % P::YB) * N + tile / P::YB, 0, 0, st.full + gg);
      }
    };
    if constexpr (G > 1)
      if (threadIdx.x == 0) issue(block_id(), 0);
    int round = 0;
    for (int tile = block_id() + g * block_count(); tile < PG::TILES; tile += G * block_count(), round++) {
      const int x = tile / P::YB, j2 = tile % P::YB;
      if constexpr (INV) {
        const int kb = 8 * ((tid >> 4) & 1), q = (tid >> 5) * 16 + (tid & 15);
        // the epilogue's rows towards L2
        if constexpr (AUX > 0) prefetch_rows<N, T>(p.aux0[b], tid, x, j2);
        if constexpr (AUX > 1) prefetch_rows<N, T>(p.aux1[b], tid, x, j2);
        if constexpr (G > 1) {
          st.wait(g, round);
          P::y_inv(buf, tw, tid, stage + kb * P::M + q, P::M,
                   [&]() { st.next(g, tid, round, [&](int gg) { issue(tile + block_count(), gg); }); });
        } else {
          P::y_inv(buf, tw, tid, src + scratch_index<N>(kb, q, j2, x), (size_t)P::M * P::YB * N, []() {});
        }
        sync();
        P::class_inv(buf, tw, tid);
        sync();
      }
      body(x, j2);
    }
    if constexpr (G > 1) {  // a wait ran out
      __syncthreads();
      if (*st.err && threadIdx.x == 0) st.drain();
      report_error(p, *st.err);
    }
  }
  // The tile is the last one of this thread's group.
  __device__ bool last(int x, int j2) const { return x * P::YB + j2 + G * block_count() >= PG::TILES; }
  // Grid reduction over the groups: arrive once acc is complete, finish at the end
  // of the kernel; fin(tot) runs in one thread.
  template <int NR, unsigned MAXM> __device__ void arrive(const KParams &p, int b, double (&acc)[NR], int *s_last) {
    group_arrive<NR, MAXM, G>(acc, red, p.partials + (size_t)b * kPartStride * kRedMax, p.tickets + b,
                              G * block_count(), block_id() + g * block_count(), g, tid, G > 1 ? N : blockDim.x,
                              s_last);
  }
  template <int NR, unsigned MAXM, class F> __device__ void finish(const KParams &p, int b, const int *s_last, F fin) {
    double tot[NR];
    if (group_finish<NR, MAXM, G>(red, p.partials + (size_t)b * kPartStride * kRedMax, p.tickets + b,
                                  G * block_count(), g, tid, G > 1 ? N : blockDim.x, s_last, tot))
      fin(tot);
  }
};

template <int N, class T> __device__ __forceinline__ void load_twiddles(const KParams &p, c2<T> *tw) {
  for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = reinterpret_cast<const c2<T> *>(p.tw)[i];
}

// Prologue of a row's points (FP32 policies with FACC sum in FP32 first).
template <class T, class Pro, int N1, class F, class ACC>
__device__ __forceinline__ void run_prologue(F &&points, ACC &acc) {
  if constexpr (use_facc<T, Pro>()) {
    float fa[Pro::NR];
    facc_init<Pro::NR, Pro::MAXM>(fa);
    points(fa);
    facc_fold<Pro::NR, Pro::MAXM>(acc, fa);
  } else {
    points(acc);
  }
}

// --------------------------------------------------------------- plane_fwd
// Real field p.in -> scratch p.out.
// Pro: static constexpr int NR; static constexpr unsigned MAXM;
//      __device__ static T2 pro(const KParams&, int b, size_t idx, T2 x, double (&acc)[NR]);
//        (x = reals idx, idx+1 of the input field; returns the values to transform)
//      __device__ static void fin(const KParams&, int b, const double (&tot)[NR]);
template <int N, class T, class Pro>
__global__ void __launch_bounds__(N, PlaneGeo<N, T>::CPS)
    plane_fwd_kernel(const __grid_constant__ KParams p) {
  using T2 = c2<T>;
  using P = Plane<N, T>;
  constexpr int N1 = P::N1, YB = P::YB;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ int s_last[1];
  PlaneLoop<N, T, false, 1> loop(smem_raw, nullptr);
  T2 *const tw = loop.tw, *const buf = loop.buf;
  load_twiddles<N, T>(p, tw);
  grid_dep_sync();
  if (p.trigger) grid_dep_trigger();
  if (flow_stopped(p, field_id())) return;
  const int tid = loop.tid, b = field_id();
  const T *src = reinterpret_cast<const T *>(p.in[b]);
  T2 *dst = reinterpret_cast<T2 *>(p.out[b]);
  double acc[Pro::NR > 0 ? Pro::NR : 1];
  acc_init<Pro::NR, Pro::MAXM>(acc);
  __syncthreads();
  loop.run(p, b, [&](int x, int j2) {
    if (const int next = x * YB + j2 + block_count(); next < PlaneGeo<N, T>::TILES) {
      prefetch_rows<N, T>(src, tid, next / YB, next % YB);
      if constexpr (AuxOf<Pro>::value > 0) prefetch_rows<N, T>(p.aux0[b], tid, next / YB, next % YB);
      if constexpr (AuxOf<Pro>::value > 1) prefetch_rows<N, T>(p.aux1[b], tid, next / YB, next % YB);
    }
    P::rows(tid, [&](int r, int jz) {
      const size_t off = ((size_t)x * N + YB * r + j2) * N;
      const T2 *row = reinterpret_cast<const T2 *>(src + off);
      T2 v[N1];
      sfor<0, N1>([&](auto J) { v[SPM_CI(J)] = ld_field(row + 8 * SPM_CI(J) + jz); });
      run_prologue<T, Pro, N1>(
          [&](auto &a) {
            sfor<0, N1>([&](auto J) {
              constexpr int j = SPM_CI(J);
              v[j] = Pro::pro(p, b, off + 2 * (8 * j + jz), v[j], a);
            });
          },
          acc);
      P::row_store_fwd(buf, r, jz, v);
    });
    if constexpr (Pro::NR > 0)
      if (loop.last(x, j2)) loop.template arrive<Pro::NR, Pro::MAXM>(p, b, acc, s_last);
    loop.sync();
    P::class_fwd(buf, tw, tid);
    loop.sync();
    P::y_fwd(buf, tw, tid, dst, x, j2);
    loop.sync();
  });
  if constexpr (Pro::NR > 0)
    loop.template finish<Pro::NR, Pro::MAXM>(p, b, s_last, [&](double (&tot)[Pro::NR]) { Pro::fin(p, b, tot); });
}

// --------------------------------------------------------------- plane_inv
// Scratch p.in -> real field p.out.
// Epi: static constexpr int NR; static constexpr unsigned MAXM;
//      __device__ static T2 epi(const KParams&, int b, size_t idx, T2 y, double (&acc)[NR]);
//        (y = unnormalised inverse transform at reals idx, idx+1; returns values to store)
//      __device__ static void fin(const KParams&, int b, const double (&tot)[NR]);
template <int N, class T, class Epi>
__global__ void __launch_bounds__(inv_groups<N, T>() * N, PlaneGeo<N, T, inv_groups<N, T>()>::CPS)
    plane_inv_kernel(const __grid_constant__ TileParams<inv_groups<N, T>()> p) {
  using T2 = c2<T>;
  using P = Plane<N, T>;
  constexpr int G = inv_groups<N, T>();
  constexpr int N1 = P::N1, YB = P::YB;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ int s_ctl[1 + G], s_last[G];  // s_ctl: the stage's error word and counts
  PlaneLoop<N, T, true, G> loop(smem_raw, s_ctl);
  T2 *const tw = loop.tw, *const buf = loop.buf;
  load_twiddles<N, T>(p, tw);
  grid_dep_sync();
  if (p.trigger) grid_dep_trigger();
  if (flow_stopped(p, field_id())) return;
  const int tid = loop.tid, b = field_id();
  T *outb = reinterpret_cast<T *>(p.out[b]);  // null: reductions only
  double acc[Epi::NR > 0 ? Epi::NR : 1];
  acc_init<Epi::NR, Epi::MAXM>(acc);
  __syncthreads();
  loop.template run<AuxOf<Epi>::value>(p, b, [&](int x, int j2) {
    P::rows(tid, [&](int r, int jz) {
      const size_t off = ((size_t)x * N + YB * r + j2) * N;
      T2 v[N1];
      P::row_load_inv(buf, r, jz, v);
      run_prologue<T, Epi, N1>(
          [&](auto &a) {
            sfor<0, N1>([&](auto J) {
              constexpr int j = SPM_CI(J);
              const T2 o = Epi::epi(p, b, off + 2 * (8 * j + jz), v[j], a);
              if (outb) reinterpret_cast<T2 *>(outb + off)[8 * j + jz] = o;
            });
          },
          acc);
    });
    loop.sync();
  });
  if constexpr (Epi::NR > 0) {
    loop.template arrive<Epi::NR, Epi::MAXM>(p, b, acc, s_last);
    loop.template finish<Epi::NR, Epi::MAXM>(p, b, s_last, [&](double (&tot)[Epi::NR]) { Epi::fin(p, b, tot); });
  }
}

// --------------------------------------------------------------- plane_inv_fwd
// Joins a step's inverse plane pass with the next step's forward one, in place
// on the scratch p.in (= p.out): the real values never leave the registers of
// the row phase (inverse N1-point transform, epilogue, prologue, forward
// transform). phi goes to memory (p.sto) only on the step where the flow stops
// (the pencil pass armed FW_PENDING): the forward half is then skipped. A chain
// of K steps is plane_fwd, K pencils, K-1 of these and one plane_inv.
template <int N, class T, class Epi, class Pro>
__global__ void __launch_bounds__(inv_groups<N, T>() * N, PlaneGeo<N, T, inv_groups<N, T>()>::CPS)
    plane_inv_fwd_kernel(const __grid_constant__ TileParams<inv_groups<N, T>()> p) {
  using T2 = c2<T>;
  using P = Plane<N, T>;
  constexpr int G = inv_groups<N, T>();
  constexpr int N1 = P::N1, YB = P::YB;
  constexpr int NE = Epi::NR, NP = Pro::NR, NA = (NE + NP > 0) ? NE + NP : 1;
  static_assert(NA <= kRedMax, "reduction count");
  constexpr unsigned MAXM = Epi::MAXM | (Pro::MAXM << NE);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ int s_ctl[1 + G], s_last[G];  // s_ctl: the stage's error word and counts
  PlaneLoop<N, T, true, G> loop(smem_raw, s_ctl);
  T2 *const tw = loop.tw, *const buf = loop.buf;
  load_twiddles<N, T>(p, tw);
  grid_dep_sync();
  if (p.trigger) grid_dep_trigger();
  // uniform over the grid: set by the pencil pass of this step, before launch
  bool stop = false;
  if (flow_state(p, field_id(), stop)) return;
  const int tid = loop.tid, b = field_id();
  T2 *dst = reinterpret_cast<T2 *>(p.out[b]);
  T *phi = reinterpret_cast<T *>(p.sto[b]);
  double acc_e[NE > 0 ? NE : 1], acc_p[NP > 0 ? NP : 1];
  acc_init<NE, Epi::MAXM>(acc_e);
  acc_init<NP, Pro::MAXM>(acc_p);
  __syncthreads();
  loop.run(p, b, [&](int x, int j2) {
    P::rows(tid, [&](int r, int jz) {
      const size_t off = ((size_t)x * N + YB * r + j2) * N;
      T2 v[N1];
      P::row_load_inv(buf, r, jz, v);
      sfor<0, N1>([&](auto J) {
        constexpr int j = SPM_CI(J);
        v[j] = Epi::epi(p, b, off + 2 * (8 * j + jz), v[j], acc_e);
      });
      if (stop) {
        sfor<0, N1>([&](auto J) { reinterpret_cast<T2 *>(phi + off)[8 * SPM_CI(J) + jz] = v[SPM_CI(J)]; });
        return;
      }
      run_prologue<T, Pro, N1>(
          [&](auto &a) {
            sfor<0, N1>([&](auto J) {
              constexpr int j = SPM_CI(J);
              v[j] = Pro::pro(p, b, off + 2 * (8 * j + jz), v[j], a);
            });
          },
          acc_p);
      P::row_store_fwd(buf, r, jz, v);
    });
    if (loop.last(x, j2)) {
      double all[NA];
#pragma unroll
      for (int r = 0; r < NE; r++) all[r] = acc_e[r];
#pragma unroll
      for (int r = 0; r < NP; r++) all[NE + r] = acc_p[r];
      if constexpr (NE + NP == 0) all[0] = 0.0;
      loop.template arrive<NA, MAXM>(p, b, all, s_last);
    }
    loop.sync();
    if (!stop) {
      P::class_fwd(buf, tw, tid);
      loop.sync();
      P::y_fwd(buf, tw, tid, dst, x, j2);
      loop.sync();
    }
  });
  if (stop) {  // u back from tile order (p.aux0) into the caller's packed spectrum (p.aux1)
    constexpr int M = Geo<N>::M;
    const T2 *ut = reinterpret_cast<const T2 *>(p.aux0[b]);
    T2 *u = reinterpret_cast<T2 *>(const_cast<void *>(p.aux1[b]));
    for (int row = block_id(); row < N * N; row += block_count()) {
      const int kx = row / N, ky = row % N;
      for (int c = threadIdx.x; c < M; c += blockDim.x)
        u[(size_t)row * M + c] = ut[state_index<N, T>(ky % 32, ky / 32, kx, c, 1)];
    }
  }
  loop.template finish<NA, MAXM>(p, b, s_last, [&](double (&tot)[NA]) {
    double te[NE > 0 ? NE : 1], tp[NP > 0 ? NP : 1];
#pragma unroll
    for (int r = 0; r < NE; r++) te[r] = tot[r];
#pragma unroll
    for (int r = 0; r < NP; r++) tp[r] = tot[NE + r];
    Epi::fin(p, b, te);
    if (!stop) Pro::fin(p, b, tp);
  });
}

// --------------------------------------------------------------- pencil
// Op: static constexpr bool FI (forward transform of the scratch p.in), SI (load
//     state p.st), SO (store state p.sto), INV (inverse transform into the
//     scratch p.out), LIN (the op acts identically on both halves of the packed
//     c = 0 column, so no unpack), SYM (the op uses the pair kernel G);
//     static constexpr int NR; static constexpr unsigned MAXM;
//     __device__ static void point(const KParams&, int b, int Kx, int Ky, int Kz,
//         double G, T2 f, T2 s, T2 &so, T2 &inv, double (&acc)[NR], double w);
//       f = unnormalised forward value, s = state value, w = multiplicity of the
//       point in the full N^3 spectrum (1 on the kz = 0, N/2 planes, else 2).
//     __device__ static void fin(const KParams&, int b, const double (&tot)[NR]);
// States are packed spectra spec[(kx N + ky) M + column], or, inside a gradient
// chain, in tile order (p.st_tiled, p.sto_tiled): 32-byte runs 2 N^2 values
// apart become contiguous tiles.
//
// A tile has three exchange-separated phases per direction:
//   thread (cc, jx, j2) : 16-point x transforms (x = M1 j1 + jx), to and from
//                         the scratch (N / 256 of the threads);
//   (cc, jx, k1x)       : two tasks of YB-point y transforms, with both
//                         twiddles (w^{j2 k1}, w^{jx k1x});
//   (cc, k1x, k2)       : M1-point x transforms; the operator on the M1 points
//                         kx = k1x + 16 k2x of (ky, column). All threads: the
//                         operator is the longest phase.
// The last two read and write the same slots, so a tile takes five barriers.
// The tiles of column group 0 hold C/2 columns of the two k1 that -ky maps to
// each other ({0, 16} or {k1, 32 - k1}), so that the partners at (-kx, -ky)
// that unpack the c = 0 column are in the tile.
template <int N, class T, class Op>
__global__ void __launch_bounds__(PencilGeo<N, T>::TH, PencilGeo<N, T>::CPS)
    pencil_kernel(const __grid_constant__ KParams p) {
  using G = Geo<N>;
  using PG = PencilGeo<N, T>;
  using T2 = c2<T>;
  __shared__ int s_last[1];
  constexpr int R = kRun;
  constexpr int M1 = G::M1, YB = G::YB, C = PG::C, TH = PG::TH, KS = PG::KS, JS = PG::JS, NCG = PG::NCG;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  T2 *tw = reinterpret_cast<T2 *>(smem_raw);
  T2 *ex = tw + N;
  double2 *gx = reinterpret_cast<double2 *>(ex + PG::UNITS + (PG::UNITS & 1));  // symbol factors per |K|
  double *red = reinterpret_cast<double *>(gx + N / 2 + 1);
  const int tid = threadIdx.x, b = field_id();
  load_twiddles<N, T>(p, tw);
  if constexpr (Op::SYM)
    for (int i = tid; i <= N / 2; i += TH) gx[i] = __ldg(gtab_of(p, b) + i);
  grid_dep_sync();
  if (p.trigger) grid_dep_trigger();
  if (flow_stopped(p, field_id())) return;
  // read once, behind the wait (volatile): a register for all points
  double pre = 0.0;
  if constexpr (PreOf<Op>::value >= 0) pre = *((volatile const double *)p.scal + b * kScal + PreOf<Op>::value);
  const int cc = tid % C;
  const int jx = (tid / C) % M1, j2 = tid / (M1 * C);  // first / last phase
  const bool has_io = j2 < YB;
  const int ka = (tid / C) % 16, kb = tid / (C * 16);  // operator phase: k1x, k2
  double acc[Op::NR > 0 ? Op::NR : 1];
  acc_init<Op::NR, Op::MAXM>(acc);
  __syncthreads();
  const T2 *src = reinterpret_cast<const T2 *>(p.in[b]);
  T2 *dst = reinterpret_cast<T2 *>(p.out[b]);
  const T2 *st = reinterpret_cast<const T2 *>(p.st[b]);
  T2 *sto = reinterpret_cast<T2 *>(p.sto[b]);

  // The 16 tiles with the packed column take longer: they go to the first
  // blocks that have one tile less than the others (last round).
  const int rem = Op::LIN ? 0 : PG::TILES % block_count();
  for (int v = block_id(); v < PG::TILES; v += block_count()) {
    int g, k1;
    if (v >= rem && v < rem + 16) {
      g = 0;
      k1 = 2 * (v - rem);
    } else {
      const int n = v < rem ? v : v - 16, i = n % (2 * NCG - 1) + 1;
      g = i % NCG;
      k1 = 2 * (n / (2 * NCG - 1)) + i / NCG;
    }
    const bool pair_tile = !Op::LIN && g == 0 && (k1 & 1) == 0;  // holds the packed column
    int col = g * C + cc;
    if (g == 0) {
      const int pair = k1 >> 1, half = k1 & 1, sel = cc / (C / 2);
      k1 = pair ? (sel ? 32 - pair : pair) : 16 * sel;
      col = half * (C / 2) + cc % (C / 2);
    }
    const size_t base = scratch_index<N>(k1, col, 0, 0);
    T2 F[M1];
    if constexpr (Op::FI) {
      if (has_io) {
        T2 v[16];
        const T2 *in = src + base + ((size_t)j2 * N + jx) * R;
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] = in[j * M1 * R];
        Dft<-1, 16, T2>::run(v);
#pragma unroll
        for (int k = 0; k < 16; k++) ex[j2 * JS + k * KS + jx * C + cc] = v[k];
      }
      __syncthreads();
#pragma unroll 1
      for (int t = 0; t < 2; t++) {
        const int e = tid + TH * t, ex_jx = (e / C) % M1, ex_k = e / (M1 * C);
        T2 *q = ex + ex_k * KS + ex_jx * C + cc;
        T2 v[YB];
        sfor<0, YB>([&](auto J) {
          constexpr int j = SPM_CI(J);
          v[j] = j ? cmul(q[j * JS], tw[j * k1]) : q[0];
        });
        Dft<-1, YB, T2>::run(v);
        const T2 w = tw[ex_jx * ex_k];
        sfor<0, YB>([&](auto K) { q[SPM_CI(K) * JS] = cmul(v[SPM_CI(K)], w); });
      }
      __syncthreads();
      sfor<0, M1>([&](auto J) { F[SPM_CI(J)] = ex[kb * JS + ka * KS + SPM_CI(J) * C + cc]; });
      Dft<-1, M1, T2>::run(F);  // F[k2x] at kx = ka + 16 k2x
    }
    const int ky = k1 + 32 * kb;
    const int Ky = wave(ky, N);
    // state addresses: s + k2x * stride (read), t + k2x * stride (written)
    const size_t s0 = state_index<N, T>(k1, kb, ka, col, p.st_tiled), ss = state_kx_stride<N, T>(p.st_tiled) * 16;
    const size_t t0 = state_index<N, T>(k1, kb, ka, col, p.sto_tiled), ts = state_kx_stride<N, T>(p.sto_tiled) * 16;
    double2 gyz = {0.0, 0.0};
    if (Op::SYM) {
      const double2 gy = gx[Ky < 0 ? -Ky : Ky], gz = gx[col];
      gyz = double2{gy.x * gz.x, gy.y + gz.y};
    }
    auto sym = [&](int Kx, double2 yz) { return SymFn{Op::SYM ? pair_symbol(gx[Kx < 0 ? -Kx : Kx], yz) : 0.0, pre}; };
    const bool packed = !Op::LIN && col == 0;
    constexpr int SG = M1 <= 8 ? M1 : M1 / 2;  // state loads in flight per thread
    constexpr bool STREAM = stream_state<N, T>();
    const uint64_t spol = STREAM ? l2_stream_policy() : 0;
    auto points = [&](auto &a) {
      if (!Op::LIN) __builtin_assume(col > 0);
#pragma unroll
      for (int h = 0; h < M1; h += SG) {
        T2 s[SG];
#pragma unroll
        for (int i = 0; i < SG; i++) {
          const T2 *q = st + s0 + (h + i) * ss;
          s[i] = !Op::SI ? T2{0, 0} : STREAM ? ld_state(q, spol) : ld_state(q);
        }
#pragma unroll
        for (int i = 0; i < SG; i++) {
          const int k = h + i, Kx = wave(ka + 16 * k, N);
          const T2 f = Op::FI ? F[k] : T2{0, 0};
          T2 o_st = {0, 0}, o_inv = {0, 0};
          Op::point(p, b, Kx, Ky, col, sym(Kx, gyz), f, s[i], o_st, o_inv, a, 2.0);
          if constexpr (Op::SO) {
            if constexpr (STREAM) st_stream(sto + t0 + k * ts, o_st, spol);
            else sto[t0 + k * ts] = o_st;
          }
          F[k] = o_inv;
        }
      }
    };
    if (!pair_tile) {
      run_prologue<T, Op, M1>(points, acc);
    } else {
      // Column 0 is unpacked into X(., ., 0) and X(., ., N/2) with its partner
      // values, and repacked. Results wait in local memory until every partner
      // value is read. (A rolled loop: 32 tiles take this path, and unrolled it
      // doubled the kernel's instructions, which then missed the instruction
      // cache.)
      T2 ks[M1], kp[M1];  // states of the points and of their partners, then the results
      const int pk1 = (32 - k1) % 32, pk = (k1 == 0) ? (YB - kb) % YB : YB - 1 - kb;  // k1, k2 of -ky
      const int pc = (k1 == 0 || k1 == 16) ? cc : (cc + C / 2) % C;                   // its lane column
      T2 *own = ex + kb * JS + ka * KS + cc;
      if constexpr (Op::FI)
#pragma unroll
        for (int k = 0; k < M1; k++) own[k * C] = F[k];
      if constexpr (Op::SI) {
#pragma unroll
        for (int k = 0; k < M1; k++) {
          const int kx = ka + 16 * k;
          ks[k] = ld_state(st + s0 + k * ss);
          kp[k] = packed ? ld_state(st + state_index<N, T>(pk1, pk, kx ? N - kx : 0, 0, p.st_tiled)) : T2{0, 0};
        }
      }
      __syncthreads();
      auto points_packed = [&](auto &a) {
        double2 gym = {0.0, 0.0};  // symbol factors at kz = N/2
        if (Op::SYM) {
          const double2 gy = gx[Ky < 0 ? -Ky : Ky], gz = gx[N / 2];
          gym = double2{gy.x * gz.x, gy.y + gz.y};
        }
#pragma unroll 4
        for (int k = 0; k < M1; k++) {
          const int kx = ka + 16 * k, Kx = wave(kx, N);
          T2 f = {0, 0}, q = {0, 0}, v = {0, 0}, w = {0, 0};
          if constexpr (Op::FI) {
            const int nk = kx ? N - kx : 0;
            f = own[k * C];
            q = ex[pk * JS + (nk % 16) * KS + (nk / 16) * C + pc];
          }
          if constexpr (Op::SI) {
            v = ks[k];
            w = kp[k];
          }
          T2 o_st = {0, 0}, o_inv = {0, 0}, o_st2 = {0, 0}, o_inv2 = {0, 0};
          if (packed) {
            const T2 f0 = {(T)0.5 * (f.x + q.x), (T)0.5 * (f.y - q.y)};
            const T2 fM = {(T)0.5 * (f.y + q.y), (T)0.5 * (q.x - f.x)};
            const T2 u0 = {(T)0.5 * (v.x + w.x), (T)0.5 * (v.y - w.y)};
            const T2 uM = {(T)0.5 * (v.y + w.y), (T)0.5 * (w.x - v.x)};
            Op::point(p, b, Kx, Ky, 0, sym(Kx, gyz), f0, u0, o_st, o_inv, a, 1.0);
            Op::point(p, b, Kx, Ky, -N / 2, sym(Kx, gym), fM, uM, o_st2, o_inv2, a, 1.0);
          } else {
            Op::point(p, b, Kx, Ky, col, sym(Kx, gyz), f, v, o_st, o_inv, a, 2.0);
          }
          ks[k] = T2{o_st.x - o_st2.y, o_st.y + o_st2.x};
          kp[k] = T2{o_inv.x - o_inv2.y, o_inv.y + o_inv2.x};
        }
      };
      run_prologue<T, Op, M1>(points_packed, acc);
      __syncthreads();  // partner values in ex and in the state are read
#pragma unroll
      for (int k = 0; k < M1; k++) {
        if constexpr (Op::SO) sto[t0 + k * ts] = ks[k];
        F[k] = kp[k];
      }
    }
    if constexpr (Op::NR > 0)
      if (v + block_count() >= PG::TILES)  // the block's last tile
        group_arrive<Op::NR, Op::MAXM, 1>(acc, red, p.partials + (size_t)b * kPartStride * kRedMax, p.tickets + b,
                                          block_count(), block_id(), 0, tid, TH, s_last);
    if constexpr (Op::INV) {
      Dft<+1, M1, T2>::run(F);
      sfor<0, M1>([&](auto J) { ex[kb * JS + ka * KS + SPM_CI(J) * C + cc] = F[SPM_CI(J)]; });
      __syncthreads();
#pragma unroll 1
      for (int t = 0; t < 2; t++) {
        const int e = tid + TH * t, ex_jx = (e / C) % M1, ex_k = e / (M1 * C);
        T2 *q = ex + ex_k * KS + ex_jx * C + cc;
        const T2 w = tw[ex_jx * ex_k];
        T2 v[YB];
        sfor<0, YB>([&](auto K) { v[SPM_CI(K)] = cmulc(q[SPM_CI(K) * JS], w); });
        Dft<+1, YB, T2>::run(v);
        sfor<0, YB>([&](auto J) {
          constexpr int j = SPM_CI(J);
          q[j * JS] = j ? cmulc(v[j], tw[j * k1]) : v[0];
        });
      }
      __syncthreads();
      if (has_io) {
        T2 v[16];
#pragma unroll
        for (int k = 0; k < 16; k++) v[k] = ex[j2 * JS + k * KS + jx * C + cc];
        Dft<+1, 16, T2>::run(v);
        T2 *o = dst + base + ((size_t)j2 * N + jx) * R;
#pragma unroll
        for (int j = 0; j < 16; j++) o[j * M1 * R] = v[j];
      }
    }
    if constexpr (Op::FI || Op::INV) __syncthreads();
  }
  if constexpr (Op::NR > 0) {
    double tot[Op::NR];
    if (group_finish<Op::NR, Op::MAXM, 1>(red, p.partials + (size_t)b * kPartStride * kRedMax, p.tickets + b,
                                          block_count(), 0, tid, TH, s_last, tot))
      Op::fin(p, b, tot);
  }
}

}  // namespace spm
