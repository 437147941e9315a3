// bhr_resident.cu -- whole SSP-RK3 or RK4 steps of a small grid in one launch.
//
// Grids up to ~300 000 points fit in the SMs' shared memory.  Advanced with
// three launches a step they are bound by launch latency and by refetching
// every tile at each stage.  Here one cooperative launch runs many steps:
// every block keeps its 64-column tile (state, u^n and the time-independent
// bb) in shared memory for the whole launch, and after each stage sends only
// the edges its neighbours' stencils reach -- 3 rows of q up and down, 4
// columns of all planes left and right.  An edge value travels as one 16-byte
// word {value, stage number} written and read with single 128-bit accesses,
// so the number says when the value beside it is the one wanted: no fence, no
// separate flag, one trip through L2 per stage.  Two inboxes alternate: a
// neighbour sends stage n+2 only after it has this block's stage n+1, which
// this block sends after it has read stage n.  q's new values need p only at
// the point itself, so a row forms and sends q first and waits for p's halo
// after that: q's edges travel while p is formed, p's while the next q is.
//
// Measured on 148 SMs, us per step (three stages), stage launches (block8n) ->
// here: 256 x 32 11.8 -> 5.1, 1024 x 64 12.7 -> 5.8, 2048 x 64 15.5 -> 9.3,
// 2048 x 96 18.9 -> 18.4, 2048 x 128 21.3 -> 20.7, 4096 x 64 20.9 -> 19.9.
// With a source (the patches of a launch's steps are built before it: 0.5 us a
// step) 512 x 32 12.6 -> 5.5, 1024 x 64 13.5 -> 6.4, 2048 x 64 16.0 -> 10.0;
// RK4 512 x 32 16.1 -> 6.5, 1024 x 64 18.2 -> 7.3, 1536 x 64 20.6 -> 10.8.
// Taller tiles with a source lose to the stage launches, which build sources
// beside the stages (2048 x 128 22.2 there, 23.7 here; 1152 x 256 23.2, 24.1),
// and RK4's z takes their shared memory: both stop at 16 rows.
// At 1024 x 64 (7-row tiles) about three quarters of the step are a lone row's
// instruction stream (latency of FP64 and shared-memory chains with 4 warps a
// scheduler), the rest waiting for edges; from 9 rows on the FP64 issue rate counts, and
// taller tiles than 32 rows do not fit.
//
// The extraction column of every step goes to a history buffer, which
// chunk_integrate_kernel and chunk_project_kernel turn into the time
// integrals and the waveform rows of all the launch's steps.
#include "bhr_device.cuh"
#include "bhr_internal.h"

#include <algorithm>
#include <mutex>

namespace bhr {
namespace {

constexpr int kResWarps = 16;
constexpr int kResThreads = 32 * kResWarps;
static_assert(kResidentMaxRows == 2 * kResWarps, "tallest tile: two rows a warp");
constexpr int kMaxPolls = 1 << 21;  // bounded wait for an edge value

// The d-th closure point beyond f1 and f2 (HighOrder/kern.cu:320-449).
__device__ __forceinline__ double extrap(const double f1, const double f2, const int d) {
  const double e1 = (4.0 * f1 - f2) * kThird;
  if (d == 1) return e1;
  const double e2 = (4.0 * e1 - f1) * kThird;
  return d == 2 ? e2 : (4.0 * e2 - e1) * kThird;
}

__device__ __forceinline__ void edge_send(ulonglong2 *slot, const double v, const unsigned long long seq) {
  asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}\n" ::"l"(slot),
               "l"(__double_as_longlong(v)), "l"(seq));
}
__device__ __forceinline__ ulonglong2 edge_load(const ulonglong2 *slot) {
  ulonglong2 r;
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}\n"
               : "=l"(r.x), "=l"(r.y)
               : "l"(slot));
  return r;
}

// Three shapes: <1, 1> a row is two warps of one column a thread (tiles of up
// to 8 rows: the chip has more warp slots than rows, and a row's latency
// counts), <2, 1> a row is one warp of two columns a thread (up to 16 rows),
// <2, 2> a warp has two rows (up to 32).
__host__ __device__ constexpr int res_rows(int cols, int rpw) { return kResWarps * rpw * cols / 2; }
// Shared memory (doubles), laid out for a shape's tallest tile R so that every
// stride is a constant: q [2 buffers][2][R + 6][WC], p [1 or 2 buffers][2][R]
// [WC] (a row of one warp is updated in place), u^n [4][R][TC], RK4's z
// [4][R][TC] and, where a warp has several rows, bb [R][WC], row factors [R]
// [RF_COUNT] and column factors [CF_TILE][TC].
__host__ __device__ constexpr int res_smem_doubles(int cols, int rpw, bool rk4) {
  const int R = res_rows(cols, rpw);
  return 4 * (R + 6) * WC + (cols == 1 ? 4 : 2) * R * WC + (rk4 ? 8 : 4) * R * TC +
         (rpw == 1 ? 0 : R * WC + R * RF_COUNT + CF_TILE * TC);
}
// A block's inbox, 16-byte words: q rows from above and below [2 planes][3]
// [TC] each, q columns from the left and the right [2 planes][rmax][4] each,
// p columns [rmax][side][2 planes][4].
__host__ __device__ constexpr int res_q_words(int rmax) { return 12 * TC + 16 * rmax; }
__host__ __device__ constexpr int res_inbox_words(int rmax) { return res_q_words(rmax) + 16 * rmax; }

// The time-independent coefficients of a thread's points of a row
// (HighOrder/kern.cu:132-158, 192-197).
template <int COLS>
struct RowCoef {
  double bb[COLS], ee[COLS], dre[COLS], dim[COLS], are[COLS], aim[COLS], vre[COLS], vim[COLS], cc[COLS], ctan;
};
// bbw: bb on the point's columns -3 .. +3 (first column's -3 first).
template <int COLS>
__device__ __forceinline__ void row_coef(RowCoef<COLS> &C, const ResidentArgs &A, const double (&bbw)[6 + COLS],
                                         const double (&cf)[CF_TILE][COLS], const double s2, const double cs,
                                         const double gth, const double ctan) {
  C.ctan = ctan * A.cy;
#pragma unroll
  for (int c = 0; c < COLS; c++) {
    const double Dt = cf[CF_DT][c], bb = bbw[3 + c];
    const double ib = rcp_nr(fma(Dt, A.a2 * s2, cf[CF_B0][c]));
    const double ee = fma(cf[CF_ATN][c], ib, bb), bti = fma(Dt, A.m4a * cs, cf[CF_BI0][c]);
    const double dbdx =
        A.cx * (45.0 * (bbw[4 + c] - bbw[2 + c]) - 9.0 * (bbw[5 + c] - bbw[1 + c]) + (bbw[6 + c] - bbw[c]));
    C.bb[c] = bb;
    C.ee[c] = ee;
    C.dre[c] = fma(-dbdx, ee, fma(-bb, cf[CF_XR][c], cf[CF_YR][c]) * ib);
    C.dim[c] = fma(-bb, bti, cf[CF_BRI][c]) * ib;
    C.are[c] = cf[CF_XR][c] * ib;
    C.aim[c] = bti * ib;
    C.vre[c] = fma(Dt, gth, cf[CF_CR0][c]) * ib;
    C.vim[c] = cf[CF_CIN][c] * ib;
    C.cc[c] = -Dt * ib;
  }
}

template <int COLS>
__device__ __forceinline__ void get(double (&v)[COLS], const double *x) {
  if constexpr (COLS == 2) {
    const double2 t = *reinterpret_cast<const double2 *>(x);
    v[0] = t.x;
    v[1] = t.y;
  } else {
    v[0] = *x;
  }
}
template <int COLS>
__device__ __forceinline__ void put(double *x, const double (&v)[COLS]) {
  if constexpr (COLS == 2) *reinterpret_cast<double2 *>(x) = make_double2(v[0], v[1]);
  else *x = v[0];
}
// The window of columns -4 .. COLS+3 around a thread's columns; its own are given.
template <int COLS>
__device__ __forceinline__ void window(double (&v)[8 + COLS], const double *x, const double (&own)[COLS]) {
#pragma unroll
  for (int j = 0; j < 8 + COLS; j += COLS) {
    if (j == 4) {
#pragma unroll
      for (int c = 0; c < COLS; c++) v[4 + c] = own[c];
    } else {
      double t[COLS];
      get<COLS>(t, x - 4 + j);
#pragma unroll
      for (int c = 0; c < COLS; c++) v[j + c] = t[c];
    }
  }
}

// A pole row from its two neighbours: extrapolated for even m (w = 1/3), zero
// for odd m (w = 0).
template <int COLS>
__device__ __forceinline__ void pole(double (&g)[COLS], const double (&g1)[COLS], const double (&g2)[COLS], const double w) {
#pragma unroll
  for (int c = 0; c < COLS; c++) g[c] = (4.0 * g1[c] - g2[c]) * w;
}

// With one row per warp a thread keeps its points' coefficients in registers
// for the whole launch; with two they are formed again each stage.  SRC: the
// solve has a particle source (each step's patch read from memory).  RK4:
// classical RK4 instead of SSP-RK3, its stages combined as the stage kernels
// combine them (one row per warp only: z takes the shared memory).
template <int COLS, int RPW, bool SRC, bool RK4>
__global__ void __launch_bounds__(kResThreads, 1) resident_kernel(const __grid_constant__ ResidentArgs A) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ int abort_flag;
  constexpr bool KEEP = RPW == 1;
  constexpr int STAGES = RK4 ? 4 : 3;
  constexpr int PBUFS = COLS == 1 ? 2 : 1;
  // q edge words a thread receives: (768 + 16 rows) / 512
  constexpr int kSlots = (12 * TC + 16 * res_rows(COLS, RPW) + kResThreads - 1) / kResThreads;
  const int lane = threadIdx.x, warp = __shfl_sync(0xffffffffu, threadIdx.y, 0), tid = warp * 32 + lane;
  const int N = A.N, M = A.M;
  const size_t NM = static_cast<size_t>(N) * M;
  const int strip = blockIdx.x % A.strips, seg = blockIdx.x / A.strips;
  const int c0 = strip * TC, b0 = 3 + seg * (M - 6) / A.segs, R = 3 + (seg + 1) * (M - 6) / A.segs - b0;
  const bool has_l = strip > 0, has_r = strip + 1 < A.strips, has_t = seg > 0, has_b = seg + 1 < A.segs;
  constexpr int RS = res_rows(COLS, RPW), qpl = (RS + 6) * WC, ppl = RS * WC;  // rows laid out, plane strides
  double *const q0 = reinterpret_cast<double *>(smem_raw), *const p0 = q0 + 4 * qpl, *const un = p0 + 2 * PBUFS * ppl,
                *const zn = un + 4 * RS * TC, *const bbs = RK4 ? zn + 4 * RS * TC : zn,
                *const rowf = bbs + RS * WC, *const colf = rowf + RS * RF_COUNT;
  const int row0 = COLS == 2 ? warp : warp >> 1;                        // this warp's first row
  const int col = COLS == 2 ? 2 * lane : 32 * (warp & 1) + lane;        // this thread's first column in the tile
  const int a0 = c0 + col, w0 = col + 4;

  // Stencil weights, with the grid scales where the coefficients lack them.
  const double d1a = 45.0 * A.cx, d1b = -9.0 * A.cx, d1c_ = A.cx;
  const double y2a = __dmul_rn(-490.0, A.cyy), y2b = __dmul_rn(270.0, A.cyy), y2c = __dmul_rn(-27.0, A.cyy),
               y2d = __dmul_rn(2.0, A.cyy);
  // The second derivative's scaled weights do not add up to zero as whole ones
  // do.  What is left of their sum (formed here without rounding) acts on f
  // itself, always the same way: it is taken out of the p equation's
  // coefficient of f, with RF_G.  Left in, the error against 80 bits grows past
  // that of the stage launches with the step count (896 x 176 1.87 times as
  // large after 120 steps, 1024 x 176 4.7 times after 332; without it 0.9).
  // Whole weights instead cost 4-5 % of a step (more spills).
  const double y2_rest = KEEP ? 0.0 : 2.0 * (0.5 * y2a + y2b + y2c + y2d);

  // ---- the tile: state with its halo, and what the coefficients are made of
  if (tid == 0) abort_flag = 0;
  for (int i = tid; i < 2 * (R + 6) * (WC / 2); i += kResThreads) {
    const int pl = i / ((R + 6) * (WC / 2)), rem = i - pl * (R + 6) * (WC / 2), j = rem / (WC / 2), w = 2 * (rem - j * (WC / 2));
    const int b = b0 - 3 + j, a = c0 - 4 + w;
    double2 v = make_double2(0.0, 0.0);
    if (a >= 0 && a < N && b >= 3 && b < M - 3) v = *reinterpret_cast<const double2 *>(A.u + pl * NM + static_cast<size_t>(b) * N + a);
    *reinterpret_cast<double2 *>(q0 + pl * qpl + j * WC + w) = v;
  }
  for (int i = tid; i < (KEEP ? 2 : 3) * R * (WC / 2); i += kResThreads) {
    const int pl = i / (R * (WC / 2)), rem = i - pl * R * (WC / 2), j = rem / (WC / 2), w = 2 * (rem - j * (WC / 2));
    const int b = b0 + j, a = c0 - 4 + w;
    double2 v = make_double2(0.0, 0.0);
    const double *src = pl < 2 ? A.u + (2 + pl) * NM : A.bb;
    if (a >= 0 && a < N) v = *reinterpret_cast<const double2 *>(src + static_cast<size_t>(b) * N + a);
    *reinterpret_cast<double2 *>((pl < 2 ? p0 + pl * ppl : bbs) + j * WC + w) = v;
  }
  if (!KEEP) {
    for (int i = tid; i < R * RF_COUNT; i += kResThreads) {
      const double v = A.rowtab[static_cast<size_t>(i % RF_COUNT) * M + b0 + i / RF_COUNT];
      rowf[i] = i % RF_COUNT == RF_G ? v + y2_rest : v;
    }
    for (int i = tid; i < CF_TILE * TC; i += kResThreads) colf[i] = A.coltab[static_cast<size_t>(i / TC) * N + c0 + i % TC];
  }
  // Stored columns, and the weight of the Kreiss-Oliger term.
  bool st[COLS];
  double kon[COLS];
#pragma unroll
  for (int c = 0; c < COLS; c++) {
    st[c] = a0 + c >= 3 && a0 + c < N - 3;
    kon[c] = (a0 + c >= 4 && a0 + c < N - 4) ? -A.cko : 0.0;
  }

  // ---- the edges.  Inbox words are numbered from A.inbox on.
  const int words = res_inbox_words(A.rmax), qwords = res_q_words(A.rmax);
  const int mine = blockIdx.x * 2 * words;
  const int left = mine - 2 * words, right = mine + 2 * words, above = mine - 2 * words * A.strips,
            below = mine + 2 * words * A.strips;
  // Where this thread's q words go in a q buffer (-1: none).
  int dst[kSlots];
#pragma unroll
  for (int n = 0; n < kSlots; n++) {
    const int i = tid + n * kResThreads;
    int d = -1;
    if (i < 12 * TC) {
      const int up = i < 6 * TC, k = up ? i : i - 6 * TC, pl = k / (3 * TC), j = (k / TC) % 3, c = k % TC;
      if (up ? has_t : has_b) d = pl * qpl + (up ? j : 3 + R + j) * WC + 4 + c;
    } else if (i < qwords) {
      const int k = i - 12 * TC, rt = k >= 8 * A.rmax, e = rt ? k - 8 * A.rmax : k;
      const int pl = e / (4 * A.rmax), r = (e / 4) % A.rmax, w = (rt ? WC - 4 : 0) + e % 4;
      if ((rt ? has_r : has_l) && r < R) d = pl * qpl + (3 + r) * WC + w;
    }
    dst[n] = d;
  }
  unsigned recv = 0;
#pragma unroll
  for (int n = 0; n < kSlots; n++) recv |= (dst[n] >= 0 ? 1u : 0u) << n;
  // This lane's p word of a row: side, plane and column of the halo (a
  // half-row warp takes its side only).
  const bool p_left = COLS == 1 ? (warp & 1) == 0 : lane < 8;
  const bool p_recv = lane < (COLS == 1 ? 8 : 16) && (p_left ? has_l : has_r);
  const int p_dst = (lane >> 2 & 1) * ppl + (p_left ? 0 : WC - 4) + (lane & 3);
  const int p_word = mine + qwords + (p_left ? 0 : 8) + (lane & 7);
  // Where this thread's edges go: its columns' side (or none).
  const bool to_l = col < 4 && has_l, to_r = col >= TC - 4 && has_r;
  const int q_side = to_l ? left + 12 * TC + 8 * A.rmax + col : right + 12 * TC + col - (TC - 4);
  const int p_side = to_l ? left + qwords + 8 + col : right + qwords + col - (TC - 4);

  // Radial-end closure of a row of two planes (HighOrder/kern.cu:412-449),
  // one plane per lane, once the warp that holds the end has written it.
  const bool close_l = !has_l && (COLS == 2 || (warp & 1) == 0), close_r = !has_r && (COLS == 2 || (warp & 1) == 1);
  auto close_ends = [&](double *base, const int stride) {
    __syncwarp();
    if (lane < 2) {
      double *row = base + lane * stride;
      if (close_l) {
        row[6] = (4.0 * row[7] - row[8]) * kThird;
        row[5] = (4.0 * row[6] - row[7]) * kThird;
        row[4] = (4.0 * row[5] - row[6]) * kThird;
      }
      if (close_r) {
        row[TC + 1] = (4.0 * row[TC] - row[TC - 1]) * kThird;
        row[TC + 2] = (4.0 * row[TC + 1] - row[TC]) * kThird;
        row[TC + 3] = (4.0 * row[TC + 2] - row[TC + 1]) * kThird;
      }
    }
  };
  const bool ends = close_l || close_r;
  __syncthreads();
  RowCoef<COLS> C;
  for (int i = 0; i < RPW; i++) {
    const int r = row0 + i * kResWarps, b = b0 + r;
    if (r >= R) break;
#pragma unroll
    for (int pl = 0; pl < 4; pl++) {
      double t[COLS];
      get<COLS>(t, (pl < 2 ? q0 + pl * qpl + (3 + r) * WC : p0 + (pl - 2) * ppl + r * WC) + w0);
      put<COLS>(un + (pl * RS + r) * TC + col, t);
    }
    if (KEEP) {
      const double *row = A.bb + static_cast<size_t>(b) * N;
      double w[6 + COLS], cf[CF_TILE][COLS];
#pragma unroll
      for (int k = 0; k < 6 + COLS; k++) w[k] = row[min(max(a0 - 3 + k, 0), N - 1)];
#pragma unroll
      for (int f = 0; f < CF_TILE; f++) get<COLS>(cf[f], A.coltab + static_cast<size_t>(f) * N + a0);
      row_coef<COLS>(C, A, w, cf, A.rowtab[static_cast<size_t>(RF_S2) * M + b], A.rowtab[static_cast<size_t>(RF_COS) * M + b],
                     A.rowtab[static_cast<size_t>(RF_G) * M + b], A.rowtab[static_cast<size_t>(RF_CTAN) * M + b]);
      // The grid scales go into the kept coefficients: the stencils have whole
      // weights (fewer operations and registers: 1024 x 64 6.1 -> 5.8 us a step).
      C.ctan /= A.cyy;
#pragma unroll
      for (int c = 0; c < COLS; c++) {
        C.cc[c] *= A.cyy;
        C.bb[c] *= A.cx;
        C.ee[c] *= A.cx;
        C.dre[c] *= A.cx;
        C.dim[c] *= A.cx;
      }
    }
    if (ends) {
      close_ends(q0 + (3 + r) * WC, qpl);
      close_ends(p0 + r * WC, ppl);
    }
  }
  __syncthreads();

  // A row's targets: word offsets of this thread's edges (-1: none), and
  // whether its theta window reaches a pole.
  struct Row {
    int up, down, side, p_side, p_word, pole;
  } T;
  auto targets = [&](const int r) {
    const int b = b0 + r;
    T.up = has_t && r < 3 ? above + 6 * TC + r * TC + col : -1;
    T.down = has_b && r >= R - 3 ? below + (r - (R - 3)) * TC + col : -1;
    T.side = to_l || to_r ? q_side + r * 4 : -1;
    T.p_side = p_side + r * 16;
    T.p_word = p_recv ? p_word + r * 16 : -1;
    T.pole = b < 6 || b >= M - 6;
  };
  if (KEEP) targets(row0);
  // This thread holds extraction column hist_col & 1 in its column hist_col >>
  // 1 (never both: of 3, 4 and of N - 4, N - 5 each lies in another pair).
  int hist_col = -1;
#pragma unroll
  for (int e = 0; e < 2; e++)
    if (A.hist != nullptr && A.ext[e] >= a0 && A.ext[e] < a0 + COLS) hist_col = 2 * (A.ext[e] - a0) + e;

  auto d1 = [&](const double (&v)[8 + COLS], const int c) {
    return KEEP ? fma(45.0, v[5 + c] - v[3 + c], fma(-9.0, v[6 + c] - v[2 + c], v[7 + c] - v[1 + c]))
                : fma(d1a, v[5 + c] - v[3 + c], fma(d1b, v[6 + c] - v[2 + c], d1c_ * (v[7 + c] - v[1 + c])));
  };
  const double pole_w = A.even_m ? kThird : 0.0;
  unsigned long long seq = A.seq;
  bool aborted = false, first = true;
  int cur = 0;  // buffer of the stage input

#pragma unroll 1
  for (int step = 0; step < A.steps; step++) {
    // The step's source patch: this thread's first column and the tile's
    // first row in it.
    int src_c = 0, src_r = 0;
    const double *patch = nullptr;
    if (SRC) {
      const int k = A.ks + step;
      src_c = a0 - __ldg(&A.recs[k].col0);
      src_r = b0 - __ldg(&A.recs[k].row0);
      patch = A.src + static_cast<size_t>(k % A.nbuf) * 2 * A.PTSX * A.PTSY;
    }
#pragma unroll
    for (int stage = 1; stage <= STAGES; stage++, seq++) {
      const bool last = stage == STAGES && step + 1 == A.steps;
      const int par = static_cast<int>(seq & 1) * words, par0 = words - par;  // this stage's words, the input's
      const double *q = q0 + cur * 2 * qpl;
      double *qn = q0 + (cur ^ 1) * 2 * qpl;
      double *p = p0 + (PBUFS == 2 ? cur * 2 * ppl : 0), *pn = p0 + (PBUFS == 2 ? (cur ^ 1) * 2 * ppl : 0);
      // The stage combination, f + dt L, (3 u^n + f + dt L)/4 and (u^n + 2 f +
      // 2 dt L)/3 (HighOrder/kern.cu:301-318, 582-620), the sums of u^n and f
      // rounded as in the stage launches.  kThird is less than 1/3, so a third
      // of a field at rest comes out low by an ulp in one of four values; with
      // the weights 3/4, 1/4, 1/3 and 2/3 on the terms one by one, in one of
      // six.  Such a difference adds up: the waveform of 1024 x 64 after 2500
      // steps was 8.7e-15 from the stage launches', like this 3.8e-16.
      // RK4: u^n + dt/2 L, u^n + dt/2 L, u^n + dt L, z + y3/3 + dt/6 L.
      const double cr = RK4 ? (stage < 3 ? 0.5 * A.dt : stage == 3 ? A.dt : A.dt / 6.0)
                            : stage == 1 ? A.dt : stage == 2 ? 0.25 * A.dt : 2.0 * kThird * A.dt;
      auto terms = [&](const double f, const double u) {
        if (stage == 1) return f;
        if (RK4) return stage == 4 ? fma(kThird, f, u) : u;
        return stage == 2 ? fma(0.75, u, 0.25 * f) : kThird * fma(2.0, f, u);
      };
      const double *us = RK4 && stage == 4 ? zn : un;
#pragma unroll 1
      for (int i = 0; i < RPW; i++) {
        const int r = row0 + i * kResWarps, b = b0 + r;
        if (r >= R) break;
        if (!KEEP) targets(r);
        // This row's p halo, asked for early.
        const ulonglong2 *p_in = A.inbox + T.p_word + par0;
        ulonglong2 pw = make_ulonglong2(0, 0);
        if (T.p_word >= 0) pw = edge_load(p_in);
        // The source at its points, likewise.
        double sv[2][COLS];
        if (SRC) {
          const int sr = src_r + r;
          const bool on = sr >= 0 && sr < A.PTSY;
#pragma unroll
          for (int c = 0; c < COLS; c++) {
            const bool in = on && src_c + c >= 0 && src_c + c < A.PTSX;
            const double *x = patch + static_cast<size_t>(sr) * A.PTSX + src_c + c;
            sv[0][c] = in ? __ldg(x) : 0.0;
            sv[1][c] = in ? __ldg(x + static_cast<size_t>(A.PTSY) * A.PTSX) : 0.0;
          }
        }
        if (!KEEP) {
          double w[6 + COLS], cf[CF_TILE][COLS];
#pragma unroll
          for (int j = 0; j < 6 + COLS; j++) w[j] = bbs[r * WC + w0 - 3 + j];
#pragma unroll
          for (int f = 0; f < CF_TILE; f++) get<COLS>(cf[f], colf + f * TC + col);
          const double *rf = rowf + r * RF_COUNT;
          row_coef<COLS>(C, A, w, cf, rf[RF_S2], rf[RF_COS], rf[RF_G], rf[RF_CTAN]);
        }
        // ---- q: its new values need p at the point only, so they are
        // formed, and their edges sent, before p's halo is waited for.
        double res[2][COLS], pc[2][COLS], o[2][COLS];
#pragma unroll
        for (int pl = 0; pl < 2; pl++) {
          double g[7][COLS], v[8 + COLS];
#pragma unroll
          for (int j = 0; j < 7; j++) get<COLS>(g[j], q + pl * qpl + (r + j) * WC + w0);
          window<COLS>(v, q + pl * qpl + (3 + r) * WC + w0, g[3]);
          get<COLS>(pc[pl], p + pl * ppl + r * WC + w0);
          // Pole rows (HighOrder/kern.cu:320-409) of a row that reaches them.
          if (T.pole && b < 6) {
            if (b == 3) pole<COLS>(g[2], g[3], g[4], pole_w);
            if (b <= 4) pole<COLS>(g[1], g[2], g[3], pole_w);
            pole<COLS>(g[0], g[1], g[2], pole_w);
          }
          if (T.pole && b >= M - 6) {
            if (b == M - 4) pole<COLS>(g[4], g[3], g[2], pole_w);
            if (b >= M - 5) pole<COLS>(g[5], g[4], g[3], pole_w);
            pole<COLS>(g[6], g[5], g[4], pole_w);
          }
          double u[COLS];
          get<COLS>(u, us + (pl * RS + r) * TC + col);
#pragma unroll
          for (int c = 0; c < COLS; c++) {
            // Theta derivatives (HighOrder/kern.cu:206-226).
            const double y1 = fma(45.0, g[4][c] - g[2][c], fma(-9.0, g[5][c] - g[1][c], g[6][c] - g[0][c]));
            const double y2 = KEEP ? fma(-490.0, g[3][c], 270.0 * (g[4][c] + g[2][c])) +
                                         fma(-27.0, g[5][c] + g[1][c], 2.0 * (g[6][c] + g[0][c]))
                                   : fma(y2a, g[3][c], y2b * (g[4][c] + g[2][c])) +
                                         fma(y2c, g[5][c] + g[1][c], y2d * (g[6][c] + g[0][c]));
            const double ll = fma(C.ctan, y1, y2), f = v[4 + c];
            // Radial derivative and dissipation (HighOrder/kern.cu:233-261).
            const double fx = d1(v, c);
            const double kd = fma(-8.0, v[7 + c] + v[1 + c], v[8 + c] + v[c]) +
                              fma(28.0, v[6 + c] + v[2 + c], fma(-56.0, v[5 + c] + v[3 + c], 70.0 * f));
            o[pl][c] = fma(cr, fma(kon[c], kd, fma(-C.bb[c], fx, pc[pl][c])), terms(f, u[c]));
            if (RK4 && stage == 2) zn[(pl * RS + r) * TC + col + c] = (f + 2.0 * o[pl][c] - u[c]) * kThird;
            // the p equation's q terms (HighOrder/kern.cu:281-296)
            if (pl == 0) {
              res[0][c] = fma(C.cc[c], ll, fma(C.dre[c], fx, C.vre[c] * f));
              res[1][c] = fma(C.dim[c], fx, C.vim[c] * f);
            } else {
              res[0][c] = fma(-C.dim[c], fx, fma(-C.vim[c], f, res[0][c]));
              res[1][c] = fma(C.cc[c], ll, fma(C.dre[c], fx, fma(C.vre[c], f, res[1][c])));
            }
          }
        }
#pragma unroll
        for (int pl = 0; pl < 2; pl++) put<COLS>(qn + pl * qpl + (3 + r) * WC + w0, o[pl]);
        if (!last) {
          if (T.up >= 0) {
            ulonglong2 *s = A.inbox + T.up + par;
#pragma unroll
            for (int e = 0; e < 2 * COLS; e++) edge_send(s + (e / COLS) * 3 * TC + e % COLS, o[e / COLS][e % COLS], seq);
          }
          if (T.down >= 0) {
            ulonglong2 *s = A.inbox + T.down + par;
#pragma unroll
            for (int e = 0; e < 2 * COLS; e++) edge_send(s + (e / COLS) * 3 * TC + e % COLS, o[e / COLS][e % COLS], seq);
          }
          if (T.side >= 0) {
            ulonglong2 *s = A.inbox + T.side + par;
#pragma unroll
            for (int e = 0; e < 2 * COLS; e++) edge_send(s + (e / COLS) * 4 * A.rmax + e % COLS, o[e / COLS][e % COLS], seq);
          }
        }
        if (stage == STAGES) {
#pragma unroll
          for (int pl = 0; pl < 2; pl++) {
            put<COLS>(un + (pl * RS + r) * TC + col, o[pl]);
            if (last) {
              double *u = A.u + pl * NM + static_cast<size_t>(b) * N + a0;
#pragma unroll
              for (int c = 0; c < COLS; c++)
                if (st[c]) u[c] = o[pl][c];
            }
          }
          if (hist_col >= 0) {
            // psi at the extraction column (or one of the two its closure is made of)
            double *h = A.hist + static_cast<size_t>(4 * step + 2 * (hist_col & 1)) * M + b;
            const bool second = COLS == 2 && hist_col >= 2;
            h[0] = second ? o[0][COLS - 1] : o[0][0];
            h[M] = second ? o[1][COLS - 1] : o[1][0];
          }
        }
        if (ends) close_ends(qn + (3 + r) * WC, qpl);

        // ---- p: its halo columns, then its new values.
        if (!first && !aborted) {
          int poll = 0;
          while (!__all_sync(0xffffffffu, T.p_word < 0 || pw.y == seq - 1) && ++poll < kMaxPolls)
            if (T.p_word >= 0 && pw.y != seq - 1) pw = edge_load(p_in);
          if (T.p_word >= 0) p[p_dst + r * WC] = __longlong_as_double(pw.x);
          if (poll == kMaxPolls) {  // a neighbour's edge did not come: no further waits, the launch ends with an error
            if (lane == 0) atomicCAS(A.err, 0, 5 /* BHR_TIMEOUT */);
            abort_flag = 1;
          }
        }
        __syncwarp();
#pragma unroll
        for (int pl = 0; pl < 2; pl++) {
          double v[8 + COLS], u[COLS];
          window<COLS>(v, p + pl * ppl + r * WC + w0, pc[pl]);
          get<COLS>(u, us + ((2 + pl) * RS + r) * TC + col);
#pragma unroll
          for (int c = 0; c < COLS; c++) {
            const double fx = d1(v, c);
            const double kd = fma(-8.0, v[7 + c] + v[1 + c], v[8 + c] + v[c]) +
                              fma(28.0, v[6 + c] + v[2 + c], fma(-56.0, v[5 + c] + v[3 + c], 70.0 * v[4 + c]));
            const double t = pl == 0 ? fma(C.are[c], pc[0][c], fma(-C.aim[c], pc[1][c], res[0][c]))
                                     : fma(C.are[c], pc[1][c], fma(C.aim[c], pc[0][c], res[1][c]));
            const double x = SRC ? t + sv[pl][c] : t;
            o[pl][c] = fma(cr, fma(C.ee[c], fx, fma(kon[c], kd, x)), terms(v[4 + c], u[c]));
            if (RK4 && stage == 2) zn[((2 + pl) * RS + r) * TC + col + c] = (v[4 + c] + 2.0 * o[pl][c] - u[c]) * kThird;
          }
        }
        if (PBUFS == 1) __syncwarp();  // the row has been read
#pragma unroll
        for (int pl = 0; pl < 2; pl++) put<COLS>(pn + pl * ppl + r * WC + w0, o[pl]);
        if (!last && T.side >= 0) {
          ulonglong2 *s = A.inbox + T.p_side + par;
#pragma unroll
          for (int e = 0; e < 2 * COLS; e++) edge_send(s + (e / COLS) * 4 + e % COLS, o[e / COLS][e % COLS], seq);
        }
        if (stage == STAGES) {
#pragma unroll
          for (int pl = 0; pl < 2; pl++) {
            put<COLS>(un + ((2 + pl) * RS + r) * TC + col, o[pl]);
            if (last) {
              double *u = A.u + (2 + pl) * NM + static_cast<size_t>(b) * N + a0;
#pragma unroll
              for (int c = 0; c < COLS; c++)
                if (st[c]) u[c] = o[pl][c];
            }
          }
        }
        if (ends) close_ends(pn + r * WC, ppl);
      }
      if (!last) {  // the q edges of this stage, sent while the neighbours' p was still being formed
        unsigned pend = aborted ? 0 : recv;
        const ulonglong2 *in = A.inbox + mine + par + tid;
        for (int poll = 0; pend != 0 && poll < kMaxPolls; poll++) {
          ulonglong2 v[kSlots];
#pragma unroll
          for (int n = 0; n < kSlots; n++)
            if (pend >> n & 1) v[n] = edge_load(in + n * kResThreads);
#pragma unroll
          for (int n = 0; n < kSlots; n++)
            if ((pend >> n & 1) && v[n].y == seq) {
              qn[dst[n]] = __longlong_as_double(v[n].x);
              pend &= ~(1u << n);
            }
        }
        if (pend != 0) {
          atomicCAS(A.err, 0, 5 /* BHR_TIMEOUT */);
          abort_flag = 1;
        }
      }
      __syncthreads();
      aborted = abort_flag != 0;
      first = false;
      cur ^= 1;
    }
  }

  // The boundary closure of the state in memory (HighOrder/kern.cu:622-753),
  // for callers that read it there: pole rows on columns 3 .. N-4, then the
  // radial ends of every row, by the blocks that hold the interior values.
  if (A.close) {
    const double *q = q0 + cur * 2 * qpl, *p = p0 + (PBUFS == 2 ? cur * 2 * ppl : 0);
    auto val = [&](int pl, int r, int w) {  // tile row r, window column w; pole rows extrapolated
      auto at = [&](int rr) { return pl < 2 ? q[pl * qpl + (3 + rr) * WC + w] : p[(pl - 2) * ppl + rr * WC + w]; };
      if (r >= 0 && r < R) return at(r);
      if (!A.even_m) return 0.0;
      return r < 0 ? extrap(at(0), at(1), -r) : extrap(at(R - 1), at(R - 2), r - R + 1);
    };
    const int rlo = has_t ? 0 : -3, rhi = has_b ? R : R + 3;
    for (int i = tid; i < 4 * (rhi - rlo) * TC; i += kResThreads) {
      const int pl = i / ((rhi - rlo) * TC), rem = i - pl * (rhi - rlo) * TC, r = rlo + rem / TC, c = rem % TC, a = c0 + c;
      double v;
      if (a >= 3 && a < N - 3) {
        if (r >= 0 && r < R) continue;
        v = val(pl, r, 4 + c);
      } else {
        const bool low = a < 3;
        v = extrap(val(pl, r, low ? 7 : TC), val(pl, r, low ? 8 : TC - 1), low ? 3 - a : a - (N - 4));
      }
      A.u[pl * NM + static_cast<size_t>(b0 + r) * N + a] = v;
    }
  }
}

// ---- the extraction of a resident launch's steps ---------------------------
// The time integrals of the steps in order (rectangle rule, HighOrder/
// body.cu:174-186), a thread per theta row, and the run counters; on output
// steps a snapshot for the projection.  The history's closure points (pole
// rows, and the column itself when it lies beyond a radial end: HighOrder/
// kern.cu:622-753) are filled in first, a thread per step and point; then the
// columns of kBatch steps are read before any is used, so that their loads
// are in flight together.
constexpr int kChunkThreads = 256;
__global__ void __launch_bounds__(kChunkThreads) chunk_integrate_kernel(const __grid_constant__ ChunkArgs A) {
  constexpr int kBatch = 16;
  grid_dependency_wait();
  launch_dependents();
  const ExtractArgs &E = A.E;
  const int M = E.M, tid = threadIdx.x, k0 = E.rs->k, row0 = E.rs->nrow, phase0 = k0 % E.Fr;
  const int steps = A.steps > 0 ? A.steps : min(E.rs->ks - k0, A.max_steps);
  auto slot = [&](const int s) { return A.hist + static_cast<size_t>(4 * (A.steps > 0 ? s : (k0 + s) % kHistSteps)) * M; };
  const int a = E.ext_col, N = E.N;
  const bool end_col = a < 3 || a >= N - 3;
  for (int i = tid; i < steps * (end_col ? 4 : 2) * 2; i += kChunkThreads) {
    const int hi = i & 1, k = i >> 1;
    double *h = end_col ? slot(k >> 2) + (k & 3) * M : slot(k >> 1) + (k & 1) * M;  // (step, column, plane)
    const double f1 = hi ? h[M - 4] : h[3], f2 = hi ? h[M - 5] : h[4];
#pragma unroll
    for (int d = 1; d <= 3; d++) h[hi ? M - 4 + d : 3 - d] = E.even_m ? extrap(f1, f2, d) : 0.0;
  }
  __syncthreads();
  if (end_col) {
    for (int i = tid; i < steps * 2 * M; i += kChunkThreads) {
      const int k = i / M;
      double *h = slot(k >> 1) + (k & 1) * M + (i - k * M);
      h[0] = extrap(h[0], h[2 * M], a < 3 ? 3 - a : a - (N - 4));
    }
    __syncthreads();
  }
  int bad = 0;
  for (int b = tid; b < M; b += kChunkThreads) {
    double ir = E.integ[b], ii = E.integ[M + b], dr = E.integ[2 * M + b], di = E.integ[3 * M + b];
    double pr[kBatch], pi[kBatch];
    int n = 0, phase = phase0;  // phase: k mod Fr
    for (int s0 = 0; s0 < steps; s0 += kBatch) {
#pragma unroll
      for (int s = 0; s < kBatch; s++) {
        const double *h = slot(min(s0 + s, steps - 1)) + b;
        pr[s] = h[0];
        pi[s] = h[M];
      }
#pragma unroll
      for (int s = 0; s < kBatch; s++) {
        if (s0 + s >= steps) break;
        if (!isfinite(pr[s]) || !isfinite(pi[s])) bad = 1;
        ir = ir + pr[s] * E.dt;
        ii = ii + pi[s] * E.dt;
        dr = dr + ir * E.dt;
        di = di + ii * E.dt;
        if (phase == 0 && static_cast<double>(k0 + s0 + s) * E.dt >= E.out_start) {
          if (row0 + n < E.max_rows) {
            double *snap = A.snap + static_cast<size_t>(4 * n) * M + b;
            snap[0] = ir;
            snap[M] = ii;
            snap[2 * M] = dr;
            snap[3 * M] = di;
            if (E.psirows != nullptr) {
              E.psirows[(2 * static_cast<size_t>(row0 + n)) * M + b] = pr[s];
              E.psirows[(2 * static_cast<size_t>(row0 + n) + 1) * M + b] = pi[s];
            }
          }
          n++;
        }
        if (++phase == E.Fr) phase = 0;
        if (s0 + s + 1 == steps) {
          E.ext[b] = pr[s];
          E.ext[M + b] = pi[s];
        }
      }
    }
    E.integ[b] = ir;
    E.integ[M + b] = ii;
    E.integ[2 * M + b] = dr;
    E.integ[3 * M + b] = di;
  }
  if (__syncthreads_or(bad) && tid == 0) atomicCAS(&E.rs->err, 0, 4 /* BHR_NAN_DETECTED */);
  if (tid == 0) {
    double t = E.rs->timer;
    int n = 0, phase = phase0;
    for (int s = 0; s < steps; s++) {
      if (phase == 0 && static_cast<double>(k0 + s) * E.dt >= E.out_start && row0 + n < E.max_rows)
        E.rows[static_cast<size_t>(row0 + n++) * 16] = t - E.Xmax;
      if (++phase == E.Fr) phase = 0;
      t = t + E.dt;
    }
    A.count[0] = row0;
    A.count[1] = n;
    E.rs->timer = t;
    E.rs->nrow = row0 + n;
    E.rs->k = k0 + steps;
    if (A.steps > 0) E.rs->ks = k0 + steps;
  }
}

// The projections and dE/dt of the launch's output rows (HighOrder/proj.c:
// 37-75, HighOrder/body.cu:174-176), a block per row.
__global__ void __launch_bounds__(kChunkThreads) chunk_project_kernel(const __grid_constant__ ChunkArgs A) {
  constexpr int kSums = 15;
  __shared__ double red[kChunkThreads / 32][kSums];
  grid_dependency_wait();
  launch_dependents();
  const ExtractArgs &E = A.E;
  const int M = E.M, tid = threadIdx.x, j = blockIdx.x;
  if (j >= A.count[1]) return;
  const double *snap = A.snap + static_cast<size_t>(4 * j) * M;
  double acc[kSums];
#pragma unroll
  for (int i = 0; i < kSums; i++) acc[i] = 0.0;
  for (int b = tid; b < M; b += kChunkThreads) {
    const double ir = snap[b], ii = snap[M + b], dr = snap[2 * M + b], di = snap[3 * M + b];
#pragma unroll
    for (int l = 0; l < 7; l++) {
      const double w = E.wproj[l * M + b];
      acc[2 * l] += w * dr;
      acc[2 * l + 1] -= w * di;
    }
    acc[14] += (ir * ir + ii * ii) * E.wdedt[b];
  }
#pragma unroll
  for (int i = 0; i < kSums; i++) {
    double v = acc[i];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if ((tid & 31) == 0) red[tid >> 5][i] = v;
  }
  __syncthreads();
  if (tid < kSums) {
    double v = 0.0;
    for (int w = 0; w < kChunkThreads / 32; w++) v += red[w][tid];
    E.rows[static_cast<size_t>(A.count[0] + j) * 16 + 1 + tid] = v;
  }
}

}  // namespace

ResidentGeom resident_geometry(int N, int M, bool rk4) {
  ResidentGeom g{};
  const int sms = device_sm_count(), rows = M - 6;
  g.strips = N / TC;
  if (g.strips > sms) return g;
  g.segs = std::max(1, std::min(sms / g.strips, rows / 3));  // a neighbour's halo comes from one tile: 3 rows at least
  g.rmax = (rows + g.segs - 1) / g.segs;
  g.ok = rows / g.segs >= 3 && g.rmax <= (rk4 ? kResidentRk4Rows : kResidentMaxRows);
  return g;
}

size_t resident_inbox_bytes(const ResidentGeom &g) {
  return static_cast<size_t>(g.strips) * g.segs * 2 * res_inbox_words(g.rmax) * 16;
}

// f(kernel, shared memory bytes) for the kernel of a shape, source and
// integrator.
template <class F>
static cudaError_t with_resident_kernel(int rmax, bool src, bool rk4, F &&f) {
  auto bytes = [&](int cols, int rpw) { return static_cast<int>(sizeof(double)) * res_smem_doubles(cols, rpw, rk4); };
  if (rmax <= res_rows(1, 1)) {
    if (rk4) return src ? f(resident_kernel<1, 1, true, true>, bytes(1, 1)) : f(resident_kernel<1, 1, false, true>, bytes(1, 1));
    return src ? f(resident_kernel<1, 1, true, false>, bytes(1, 1)) : f(resident_kernel<1, 1, false, false>, bytes(1, 1));
  }
  if (rmax <= res_rows(2, 1)) {
    if (rk4) return src ? f(resident_kernel<2, 1, true, true>, bytes(2, 1)) : f(resident_kernel<2, 1, false, true>, bytes(2, 1));
    return src ? f(resident_kernel<2, 1, true, false>, bytes(2, 1)) : f(resident_kernel<2, 1, false, false>, bytes(2, 1));
  }
  if (src || rk4 || rmax > kResidentMaxRows) return cudaErrorInvalidValue;
  return f(resident_kernel<2, 2, false, false>, bytes(2, 2));
}

cudaError_t prepare_resident_kernels() {
  for (int rmax : {res_rows(1, 1), res_rows(2, 1), res_rows(2, 2)})
    for (int v = 0; v < (rmax <= res_rows(2, 1) ? 4 : 1); v++)
      if (cudaError_t e = with_resident_kernel(rmax, v & 1, v >> 1, [](auto kernel, int bytes) {
            return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
          }))
        return e;
  return cudaSuccess;
}

// A resident launch holds its SMs until its last block ends, and its blocks
// wait for one another, so launches of different streams on one device are
// put one after another (each waits for the event behind the one before).
// Beside other work no block waits for one that has not begun: the blocks of a
// cooperative launch start together, when all of them have room (with one SM
// held by another kernel for 20 ms all started after it, within a microsecond),
// and nothing that waits to start goes in before them (beside three streams of
// launches that never leave an SM idle, tiles of 8-30 us, each of eight
// launches began 30 us after the one before).
static cudaError_t launch_cooperative(void (*kernel)(const ResidentArgs), const ResidentArgs &a, size_t smem,
                                      cudaStream_t st) {
  struct Last {
    cudaEvent_t done = nullptr;
    cudaStream_t stream = nullptr;
    bool any = false;
  };
  static std::mutex mu;
  static Last last[64];
  int dev = 0;
  cudaError_t e;
  if ((e = cudaGetDevice(&dev))) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(mu);
  Last &L = last[dev];
  if (!L.done && (e = cudaEventCreateWithFlags(&L.done, cudaEventDisableTiming))) return e;
  if (L.any && L.stream != st && (e = cudaStreamWaitEvent(st, L.done, 0))) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.strips * a.segs);
  cfg.blockDim = dim3(32, kResWarps);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if ((e = cudaLaunchKernelEx(&cfg, kernel, a))) return e;
  L.any = true;
  L.stream = st;
  return cudaEventRecord(L.done, st);
}

cudaError_t launch_resident(const ResidentArgs &a, cudaStream_t st) {
  if (a.steps <= 0) return cudaSuccess;
  return with_resident_kernel(a.rmax, a.src != nullptr, a.rk4 != 0,
                              [&](auto kernel, int bytes) { return launch_cooperative(kernel, a, bytes, st); });
}

cudaError_t launch_chunk_extract(const ChunkArgs &a, cudaStream_t st) {
  cudaError_t e = launch_pdl(chunk_integrate_kernel, dim3(1), dim3(kChunkThreads), 0, st, a);
  if (e != cudaSuccess) return e;
  return launch_pdl(chunk_project_kernel, dim3(a.max_steps / a.E.Fr + 1), dim3(kChunkThreads), 0, st, a);
}

}  // namespace bhr
