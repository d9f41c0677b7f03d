// tile3d.cuh -- the 3-D tile sweep: each CTA sweeps a BX x BY x BZ brick of
// the grid held whole in shared memory, hyperplane by hyperplane.
//
// The reference sweeps one hyperplane x+y+z = level of the whole grid per
// kernel launch (single_gpu_cuda/src/phi3D_fsm.cu:161-185,
// mpi_openacc/src/phi3D_fsm.c:92-117).  Any topological order of an
// ordering's dependency DAG gives the same result (each node reads the new
// values of its three upwind neighbours and the old values of its three
// downwind ones), so this kernel cuts the grid into bricks and orders them
// twice over:
//   * inside a brick, level by level: thread (lx, ly) -- brick-local
//     coordinates in sweep order -- updates node (lx, ly, L - lx - ly) at
//     level L, from the previous level's results and the next level's old
//     values in the shared-memory copy of the brick; one barrier a level.
//     Columns are listed by diagonal lx + ly, so that a warp has a node to update
//     on BZ + 2 to BZ + 7 levels;
//   * across bricks, face by face: the threads on a brick's three downwind
//     faces write their nodes' final values to a mailbox in global memory, each
//     tagged with the sweep's epoch in one 64-bit word (a 64-bit store is
//     single-copy atomic, so a reader that sees the tag sees the value: no
//     fence, no counter).  A helper warp of the downwind brick polls those words,
//     patches the values into the upwind halo of the brick's box and arrives on
//     an mbarrier for every GL levels whose faces are there, so a brick runs some
//     16 levels and an L2 round trip behind its upwind neighbours instead of a
//     whole brick.  Persistent CTAs take bricks by ticket in wavefront order
//     (every upwind brick holds a smaller ticket), so the wait always ends.
//
// What bounds it: the dependency chain.  Waiting for whole upwind bricks makes
// a sweep (n/BX + n/BY + n/BZ) bricks of BX + BY + BZ - 2 levels deep, about 9n
// levels; handing faces over level by level brings that to the sweep's own 3n
// plus an L2 round trip per brick crossed.
// Measured (octant rounds; FP32 full round / FP32 masked round / pair round): with
// bricks that waited for whole upwind bricks, 768^3 22.0 / 13.0 / 20.5 ms, 320 x
// 300 x 280 5.3 / 3.2 / 5.5 ms; handed over level by level, 22.1 / 8.5 / 15.1 and
// 2.55 / 0.95 / 1.7 ms (23.6 / 9.5 / 16.7 and 3.15 / 1.1 / 2.2 while the helper
// looked at the abort flag between its polls, tested every level's bits on its own
// and z faces left at a brick's end).  The 768^3 full round, which has bricks
// enough to fill the chip, gains nothing from the shorter chain (issue slots are
// 56 % busy there).  Tried on the way: the helper stepping
// through the levels' barrier (29.8 ms for the 768^3 full round), a second
// helper warp sending the faces (27.9: 48 registers a thread, and the sender's
// path was the level's), warps chained by mbarriers instead of a barrier a
// level (34.4).
//
// A brick's old values do not depend on its upwind bricks, so its whole box
// (the brick and a one-node halo, rows rounded up to 16 bytes) is requested
// by one TMA copy as soon as the ticket is taken.  A neighbour cannot
// overwrite a value this brick still needs: a node next to one of this brick's
// updated nodes waits for that node's mail, which is written after this
// brick's box has landed.  New values stay in the box; the rows with a changed
// node go to global memory at the brick's end, a row at a time (a store per
// node as it is computed touches up to 32 lines a warp).
//
// MAIL false (tile3d_flags.cu): a brick waits for its visited upwind bricks to finish
// the sweep, by flag, and its box's copy brings their new values.  For contexts whose
// device has no room for mailboxes (3 bytes a node for 64-bit values on 16 x 16 x 16
// bricks, 5 on 8 x 8 x 16).
//
// Every wait is bounded (SweepArgs::wait_cycles): on expiry the kernel
// records DEV_ERR_TIMEOUT, raises the abort flag, lets its own TMA copy land
// and returns.
#pragma once
#include "god64.cuh"
#include "oct_wait.h"
#include "sweep.cuh"

namespace pdfs {

template <class T, int BX_, int BY_, int BZ, int GL_ = 4>
struct T3Geo {
  static constexpr int BX = BX_, BY = BY_;
  // box row: x0-1 .. x0+BX, rounded up to 16 bytes; the field's index has no
  // x offset, so x0 - 1 = BX*bi starts the row on a 16-byte boundary
  static constexpr int W = (int)((((BX + 2) * sizeof(T)) + 15) / 16 * 16 / sizeof(T));
  static constexpr int RY = BY + 2;       // box rows: y0-1 .. y0+BY
  static constexpr int RZ = BZ + 2;       // box planes: z0-1 .. z0+BZ
  static constexpr int PL = RY * W;       // plane stride in shared memory
  static constexpr int NL = BX + BY + BZ - 2;  // levels of one brick
  static constexpr int NC = BX * BY;      // compute threads: one per (x, y) of the brick
  static constexpr int NT = NC + 32;      // and a helper warp
  static constexpr int WV = (int)sizeof(T) / 4;  // mailbox words per value (32 value bits each)
  // mailbox of a brick: x face [(lz + ly) % BZ][ly], y face [(lz + lx) % BZ][lx],
  // z face [(lx + ly) % BY][lx] -- one row per level of the reading brick, and
  // (the modulus) no unused entries
  static constexpr int MX = 0, MY = BZ * BY, MZ = MY + BZ * BX, MAIL = MZ + BX * BY;
  static constexpr int GL = GL_;  // levels handed over together
  static constexpr int SL = GL < (sizeof(T) == 4 ? 4 : 2) ? GL : sizeof(T) == 4 ? 4 : 2;  // levels polled at a time
  static constexpr int NBX = BX / 8, NBY = BY / 8, NZB = BZ / 8;  // 8^3 scheduler blocks per brick
  static constexpr int NB = NBX * NBY * NZB;
  static constexpr unsigned BOX_BYTES = (unsigned)(W * RY * RZ * sizeof(T));
  static constexpr size_t OFF_MASK = ((size_t)BOX_BYTES + 127) & ~size_t(127);
  using PlaneBits = typename std::conditional<(BZ > 32), unsigned long long, unsigned>::type;  // one bit per plane
  static constexpr size_t OFF_CHG = OFF_MASK + (size_t)BZ * BY * 4;
  static constexpr size_t OFF_BAR = OFF_CHG + (size_t)NC * sizeof(PlaneBits);
  // the box's barrier, then one per GL levels (their upwind faces are there)
  static constexpr int NG = (NL + GL - 1) / GL;
  static constexpr size_t BYTES = OFF_BAR + 8 + (size_t)NG * 8;
  // resident CTAs asked of the compiler: what shared memory allows, at most 4
  // (56 registers a thread: 3 CTAs with more cost the 768^3 rounds 4 to 9 %)
  static constexpr int CTAS = 227 * 1024 / (int)(BYTES + 1536) < 4 ? 227 * 1024 / (int)(BYTES + 1536) : 4;
  using LevelBits = typename std::conditional<(NL > 64), unsigned __int128, unsigned long long>::type;  // one bit per level
  __device__ static __forceinline__ int top(LevelBits b) {  // one past the highest bit
    const unsigned long long lo = (unsigned long long)b;
    if constexpr (sizeof(LevelBits) == 16) {
      const unsigned long long hi = (unsigned long long)(b >> 64);
      if (hi) return 128 - __clzll((long long)hi);
    }
    return lo ? 64 - __clzll((long long)lo) : 0;
  }
  // a column's planes as bits: sweep order <-> grid order
  __device__ static __forceinline__ PlaneBits flip(PlaneBits b) {
    if constexpr (BZ > 32)
      return __brevll(b) >> (64 - BZ);
    else
      return __brev(b) >> (32 - BZ);
  }
  // bits [s, s + 32) of the planes (s may be negative), and back
  __device__ static __forceinline__ unsigned level_word(PlaneBits b, int s) {
    const unsigned long long w = b;
    return s >= 64 || s <= -64 ? 0u : (unsigned)(s >= 0 ? w >> s : w << -s);
  }
  __device__ static __forceinline__ PlaneBits plane_bits(unsigned w, int s) {
    const unsigned long long v = w;
    return s >= 64 || s <= -64 ? PlaneBits(0) : PlaneBits(s >= 0 ? v << s : v >> -s);
  }
  static_assert(BZ % 8 == 0 && BY % 8 == 0 && BX % 8 == 0, "bricks hold whole 8^3 blocks");
  static_assert(BX <= BZ && BY <= BZ, "x and y mailbox rows wrap at most once");
  static_assert(BX + BY <= 32 && NB <= 32 && NZB * (NBX + NBY) + NBX * NBY <= 32, "one lane each");
  static_assert((W * sizeof(T)) % 16 == 0, "TMA rows are 16-byte multiples");
};

// FP64 reference and fast arithmetic: the solvers of god64.cuh.
template <class T, int ARITH>
constexpr bool kGod64Of = sizeof(T) == 8 && (ARITH == ARITH_REF || ARITH == ARITH_FAST);

// Their faces go over after every level (64^3 / 384^3 reference sweeps in 8 x 8 x 16
// bricks, all else equal: 953 us and 12.2 ms; in groups of 2, 1128 and 12.9; of 4,
// 1292 and 13.4): a level is 2000 to 4000 cycles, more than an L2 round trip.  An
// FP32 or pair level is 200 to 300: groups of 4 (of 2: 7 to 15 % faster on FP32
// grids to 64^3, 7 % slower at 768^3 and for pairs).
template <class T, int BX, int BY, int BZ, int ARITH>
using T3GeoOf = T3Geo<T, BX, BY, BZ, kGod64Of<T, ARITH> ? 1 : 4>;

// The levels' barrier: the compute threads.
template <int N>
__device__ __forceinline__ void level_bar() {
  asm volatile("bar.sync 1, %0;\n" ::"n"(N) : "memory");
}

// One ticket, decoded (shared memory; two slots, the next ticket's is filled
// while a brick runs).
struct T3Desc {
  int stop;          // no ticket left, or the kernel is giving up
  int li, lj, lk;    // the brick in sweep order
  int sx, sy, sz;    // the sweep's directions
  int sweep;         // OCT: which sweep of the round
  int tile, epoch;   // the brick in grid order; the sweep's flag value and mail tag
  unsigned long long *mail;  // the brick's mailbox
  int lev0, lev1;    // its levels [lev0, lev1): those that reach its visited planes
  // visited 8^3 blocks, one bit each: the brick's own (z, y, x; x fastest), and
  // the ones across its upwind faces (x: z, y; y: z, x; z: y, x)
  unsigned act, upx, upy, upz;
};

// The brick's BX x BY columns are listed by diagonal d = lx + ly (then by
// ly).  Column (lx, ly) holds a node of level L
// for L - lx - ly in [0, BZ), so a warp whose 32 columns span diagonals
// d0 .. d1 runs the level body on BZ + d1 - d0 levels: BZ + 2 to BZ + 7 for
// 16 x 16 columns listed by diagonal, BZ + 16 for the row-major warp of two
// rows (158 against 256 warp-level bodies per 16^3 brick).
template <int BX, int BY>
__device__ __forceinline__ int diag_rank(int lx, int ly) {  // the position of column (lx, ly) in that order
  constexpr int S = BX < BY ? BX : BY, M = BX < BY ? BY : BX;
  const int d = lx + ly, t = BX + BY - 1 - d;
  const int before = d <= S ? d * (d + 1) / 2 : d <= M ? S * (S + 1) / 2 + (d - S) * S : BX * BY - t * (t + 1) / 2;
  return before + ly - max(0, d - (BX - 1));
}

// The ticket taken next, decoded into d by one warp.  Tickets of bricks
// without a visited block are passed over (no brick waits for them).  In a
// round, the brick and its six face neighbours have to finish their latest
// earlier sweep first: lanes 0..6 leave in wait_flag a flag that is not there
// yet (else -1), for t3_wait once the current brick has published its own.  Without
// mail lanes 7..9 do so for the visited upwind bricks of this sweep.
template <class G, bool OCT, bool MAIL>
__device__ __forceinline__ void t3_next(const SweepArgs &a, int ntile, T3Desc &d, volatile int *s_abort,
                                        int &wait_flag, int &wait_epoch) {
  const int lane = threadIdx.x & 31;
  const int ntx = a.ntx, nty = a.nty, ntz = a.ntz;
  wait_flag = -1;
  for (;;) {
    int tk = 0;
    if (lane == 0) tk = (*s_abort || *(volatile int *)(a.err + 1)) ? ntile : atomicAdd(a.ticket, 1);
    tk = __shfl_sync(0xffffffffu, tk, 0);
    if (tk >= ntile) {
      if (lane == 0) d.stop = 1;
      break;
    }
    int lt = __ldg(a.torder + tk), osw = 0;  // OCT: (sweep << 27) | brick, else the brick, in sweep order
    int sx = a.sx, sy = a.sy, sz = a.sz;
    unsigned obit = 0;   // OCT: the ordering's bit
    bool every = false;  // the sweep visits every block
    if constexpr (OCT) {
      osw = lt >> 27;
      lt &= 0x07ffffff;
      const int sn = (a.oct_first + osw) % 8 + 1;
      obit = 1u << (sn - 1);
      every = (a.oct_full >> osw) & 1u;
      ordering_signs(sn, &sx, &sy, &sz);
    } else {
      every = a.blk_active == nullptr;
    }
    const int li = lt % ntx, lj = (lt / ntx) % nty, lk = lt / (ntx * nty);
    const int bi = sx > 0 ? li : ntx - 1 - li, bj = sy > 0 ? lj : nty - 1 - lj, bk = sz > 0 ? lk : ntz - 1 - lk;
    const int tile = (bk * nty + bj) * ntx + bi;
    const int bx0 = G::NBX * bi, by0 = G::NBY * bj, bz0 = G::NZB * bk;  // the brick's first block
    auto visited = [&](int bx, int by, int bz) -> bool {
      if (bx < 0 || by < 0 || bz < 0 || bx >= a.nbx || by >= a.nby || bz >= a.nbz) return false;
      const long long b = ((long long)bz * a.nby + by) * a.nbx + bx;
      if constexpr (OCT)
        return every || (__ldg(a.oct_bits + b) & obit) != 0;
      else
        return every || __ldg(a.blk_active + b) != 0;
    };
    bool on = false;
    if (lane < G::NB)
      on = visited(bx0 + lane % G::NBX, by0 + (lane / G::NBX) % G::NBY, bz0 + lane / (G::NBX * G::NBY));
    const unsigned act = __ballot_sync(0xffffffffu, on);
    if (act == 0) continue;
    constexpr int UX = G::NBY * G::NZB, UY = G::NBX * G::NZB, UZ = G::NBX * G::NBY;
    on = false;
    if (lane < UX) {
      on = li > 0 && visited(sx > 0 ? bx0 - 1 : bx0 + G::NBX, by0 + lane % G::NBY, bz0 + lane / G::NBY);
    } else if (lane < UX + UY) {
      const int i = lane - UX;
      on = lj > 0 && visited(bx0 + i % G::NBX, sy > 0 ? by0 - 1 : by0 + G::NBY, bz0 + i / G::NBX);
    } else if (lane < UX + UY + UZ) {
      const int i = lane - UX - UY;
      on = lk > 0 && visited(bx0 + i % G::NBX, by0 + i / G::NBX, sz > 0 ? bz0 - 1 : bz0 + G::NZB);
    }
    const unsigned up = MAIL ? __ballot_sync(0xffffffffu, on) : 0u;
    if constexpr (OCT) {
      // the round's earlier sweeps, lanes 0..6: the brick, then its neighbours
      if (lane < 7) {
        int n = -1;
        if (lane == 0) n = tile;
        if (lane == 1 && bi > 0) n = tile - 1;
        if (lane == 2 && bi < ntx - 1) n = tile + 1;
        if (lane == 3 && bj > 0) n = tile - ntx;
        if (lane == 4 && bj < nty - 1) n = tile + ntx;
        if (lane == 5 && bk > 0) n = tile - ntx * nty;
        if (lane == 6 && bk < ntz - 1) n = tile + ntx * nty;
        const int need = n >= 0 ? oct_latest(osw, a.oct_first, a.oct_full, a.oct_tbits, n) : -1;
        // (the CTA's current brick may be among them: looked at here, waited for later)
        if (need >= 0 && ld_acquire_gpu(a.tflag + n) < a.epoch + need) {
          wait_flag = n;
          wait_epoch = a.epoch + need;
        }
      }
      __syncwarp();
    }
    if constexpr (!MAIL) {
      if (lane >= 7 && lane < 10) {
        const int n = lane == 7   ? (li > 0 ? tile - sx : -1)
                      : lane == 8 ? (lj > 0 ? tile - sy * ntx : -1)
                                  : (lk > 0 ? tile - sz * ntx * nty : -1);
        const int epoch = OCT ? a.epoch + osw : a.epoch;
        bool want = n >= 0;
        if (want && !every) want = OCT ? (__ldg(a.oct_tbits + n) & obit) != 0 : __ldg(a.tact + n) != 0;
        if (want && ld_acquire_gpu(a.tflag + n) < epoch) {
          wait_flag = n;
          wait_epoch = epoch;
        }
      }
      __syncwarp();
    }
    if (lane == 0) {
      // the planes of the brick's visited blocks, in sweep order
      unsigned zb = 0;
#pragma unroll
      for (int q = 0; q < G::NZB; ++q)
        if ((act >> (q * UZ)) & ((1u << UZ) - 1u)) zb |= 1u << q;
      const int q0 = __ffs(zb) - 1, q1 = 31 - __clz(zb);
      const int lo = sz > 0 ? 8 * q0 : 8 * (G::NZB - 1 - q1), hi = sz > 0 ? 8 * q1 + 7 : 8 * (G::NZB - 1 - q0) + 7;
      d.stop = 0;
      d.li = li;
      d.lj = lj;
      d.lk = lk;
      d.sx = sx;
      d.sy = sy;
      d.sz = sz;
      d.sweep = osw;
      d.tile = tile;
      d.epoch = OCT ? a.epoch + osw : a.epoch;
      d.mail = a.pmail + (size_t)tile * (G::MAIL * G::WV);
      d.lev0 = lo;                                    // column (0, 0) reaches the first visited plane
      d.lev1 = min(G::NL, hi + G::BX + G::BY - 1);    // the last column leaves the last one
      d.act = act;
      d.upx = up & ((1u << UX) - 1u);
      d.upy = (up >> UX) & ((1u << UY) - 1u);
      d.upz = (up >> (UX + UY)) & ((1u << UZ) - 1u);
    }
    break;
  }
  __syncwarp();
}

// Waits (bounded) for the flag that t3_next left.
__device__ __forceinline__ void t3_wait(const SweepArgs &a, int wait_flag, int wait_epoch, volatile int *s_abort) {
  if (wait_flag >= 0 && ld_acquire_gpu(a.tflag + wait_flag) < wait_epoch) {
    const long long t0 = cycles();
    unsigned nap = 32;
    while (ld_acquire_gpu(a.tflag + wait_flag) < wait_epoch) {
      if (*s_abort || *(volatile int *)(a.err + 1)) {
        *s_abort = 1;
        break;
      }
      if (cycles() - t0 > a.wait_cycles) {
        raise_timeout(a, wait_flag, s_abort);
        break;
      }
      __nanosleep(nap);
      nap = min(nap * 2, 256u);
    }
  }
  __syncwarp();
}

// A mailbox entry as loaded: a tagged word per 32 value bits.
template <class T>
struct Mail {
  unsigned long long w[sizeof(T) / 4];
  __device__ __forceinline__ void load(const unsigned long long *e) {
    if constexpr (sizeof(T) == 4)
      w[0] = ld_relaxed_gpu_u64(e);
    else
      asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];\n" : "=l"(w[0]), "=l"(w[1]) : "l"(e) : "memory");
  }
  __device__ __forceinline__ bool tagged(int epoch) const {
    bool ok = (unsigned)(w[0] >> 32) == (unsigned)epoch;
    if constexpr (sizeof(T) == 8) ok = ok && (unsigned)(w[1] >> 32) == (unsigned)epoch;
    return ok;
  }
  __device__ __forceinline__ T value() const {
    if constexpr (sizeof(T) == 4)
      return __uint_as_float((unsigned)w[0]);
    else
      return __hiloint2double((int)(unsigned)w[1], (int)(unsigned)w[0]);
  }
};

// The helper's receiving: lanes [0, BY) the x-face rows and [BY, BY + BX)
// the y-face columns, and (a second set) lanes [0, BX) the z-face columns.  A
// lane reads position p of its row or column k at level k + p: p runs along z
// for the x and y faces, along y for the z face.  It polls SL levels at a time,
// as far ahead of the compute warps as the mail is there, patches the values
// into the box and arrives on the barrier of each group of GL levels.  Mail is
// awaited where the upwind brick's 8^3 block and mine are both visited: other
// halo values are the box's own.
template <class T, class G>
__device__ __forceinline__ void t3_receive(const SweepArgs &a, const T3Desc &d, int tile, int epoch, T *box, int x0,
                                           int y0, int zcnt, uint64_t *grp, volatile int *s_abort) {
  constexpr int BX = G::BX, BY = G::BY, BZ = G::NZB * 8, W = G::W, PL = G::PL;
  using LevelBits = typename G::LevelBits;
  const int lane = threadIdx.x & 31;
  const bool px = d.sx > 0, py = d.sy > 0, pz = d.sz > 0;
  const bool xf = lane < BY, yf = !xf && lane < BY + BX;
  const int k = xf ? lane : lane - BY;
  const int ku = xf ? (py ? k : BY - 1 - k) : (px ? k : BX - 1 - k), zu = px ? lane : BX - 1 - lane;  // in grid order
  // awaited levels, one bit each
  LevelBits nf = 0, nz = 0;
  if (xf ? d.li > 0 && y0 + ku <= a.ny : yf && d.lj > 0 && x0 + ku <= a.nx) {
#pragma unroll
    for (int q = 0; q < G::NZB; ++q) {
      const int c8 = min(8, zcnt - 8 * q);
      if (c8 <= 0) break;
      const unsigned mine = xf ? d.act >> ((q * G::NBY + (ku >> 3)) * G::NBX + (px ? 0 : G::NBX - 1))
                               : d.act >> ((q * G::NBY + (py ? 0 : G::NBY - 1)) * G::NBX + (ku >> 3));
      const unsigned theirs = xf ? d.upx >> (q * G::NBY + (ku >> 3)) : d.upy >> (q * G::NBX + (ku >> 3));
      if (mine & theirs & 1u) nf |= LevelBits((1u << c8) - 1u) << (k + (pz ? 8 * q : BZ - 8 * q - c8));
    }
  }
  if (lane < BX && d.lk > 0 && x0 + zu <= a.nx) {
#pragma unroll
    for (int q = 0; q < G::NBY; ++q) {
      const int c8 = min(8, a.ny - y0 + 1 - 8 * q);
      if (c8 <= 0) break;
      const unsigned mine = d.act >> (((pz ? 0 : G::NZB - 1) * G::NBY + q) * G::NBX + (zu >> 3));
      if (mine & (d.upz >> (q * G::NBX + (zu >> 3))) & 1u)
        nz |= LevelBits((1u << c8) - 1u) << (lane + (py ? 8 * q : BY - 8 * q - c8));
    }
  }
  // past the last awaited level every level is ready
  const int gend = min(d.lev1, __reduce_max_sync(0xffffffffu, max(G::top(nf), G::top(nz))));
  // mail of level lv: row lv (mod the face's rows) of the upwind brick's face
  const long long upf = xf ? tile - d.sx : tile - d.sy * a.ntx, upz = tile - d.sz * a.ntx * a.nty;
  const unsigned long long *mf = a.pmail + (upf * G::MAIL + (xf ? G::MX : G::MY) + k) * G::WV;
  const unsigned long long *mz = a.pmail + (upz * G::MAIL + G::MZ + lane) * G::WV;
  const int fcols = BX == BY ? BX * G::WV : (xf ? BY : BX) * G::WV;
  // box element read at level 0 and the step per level
  const int fs = pz ? PL : -PL, zs = py ? W : -W;
  T *bf = box + (pz ? 1 : BZ) * PL + (xf ? (1 + ku) * W + (px ? 0 : BX + 1) : (py ? 0 : BY + 1) * W + 1 + ku) - k * fs;
  T *bz = box + (pz ? 0 : BZ + 1) * PL + (py ? 1 : BY) * W + 1 + zu - lane * zs;
  constexpr int GL = G::GL, SL = G::SL;
  static_assert(BZ % GL == 0 && BY % GL == 0 && GL % SL == 0, "a group's rows are consecutive");
  bool live = true;  // false: gave up; the compute threads run out their levels (the call returns an error)
  for (int g = 0; g < G::NG; ++g) {
    if (g * GL < gend && live) {
#pragma unroll 1
      for (int L = g * GL; L < g * GL + GL; L += SL) {
        const unsigned wf = (unsigned)(nf >> L) & ((1u << SL) - 1u);  // awaited: level L + i
        const unsigned wz = L < BX + BY - 1 ? (unsigned)(nz >> L) & ((1u << SL) - 1u) : 0u;
        const unsigned long long *pf = mf + (L >= BZ ? L - BZ : L) * fcols, *pzm = mz + (L % BY) * (BX * G::WV);
        Mail<T> v[SL], w[SL];
        const long long t_last = cycles();
        unsigned nap = 0;
        for (int tries = 0;; ++tries) {
#pragma unroll
          for (int i = 0; i < SL; ++i) {  // all the loads first: they are in flight together
            if (wf & (1u << i)) v[i].load(pf + i * fcols);
            if (wz & (1u << i)) w[i].load(pzm + i * (BX * G::WV));
          }
          bool ok = true;
#pragma unroll
          for (int i = 0; i < SL; ++i) {
            if (wf & (1u << i)) ok = ok && v[i].tagged(epoch);
            if (wz & (1u << i)) ok = ok && w[i].tagged(epoch);
          }
          if (__all_sync(0xffffffffu, ok)) break;
          // a poll is a round trip to L2: the first ones follow on one another (looking
          // at the abort flag in between is another round trip on the sweep's chain)
          if (tries >= 16 && helper_idle(a, tile, s_abort, t_last, nap)) {
            live = false;
            break;
          }
        }
#pragma unroll
        for (int i = 0; i < SL; ++i) {
          if (wf & (1u << i)) bf[(L + i) * fs] = v[i].value();
          if (wz & (1u << i)) bz[(L + i) * zs] = w[i].value();
        }
        __syncwarp();
      }
    }
    if (lane == 0) mbar_arrive(grp + g);
  }
}

// OCT: an octant round -- up to kOctMax sweeps in one launch (a cycle of the
// 8 orderings).  A ticket names (sweep j, brick); ordering (oct_first + j) % 8 + 1
// visits the bricks and blocks whose bits name it, or every brick when bit j
// of oct_full is set.  Before its box is read, a brick waits until it and its six face neighbours have finished their latest
// earlier sweep of the round (their values are this sweep's old values); its
// upwind faces of this sweep come by mail as usual.  Flags carry epoch + j, so
// "finished sweep j" is a flag >= epoch + j; the ticket list (k_oct_plan,
// k_oct_merge) interleaves the sweeps by wavefront level with every brick
// after the ones it waits on, so every wait is on a smaller ticket.  The
// result is the sequential sweeps', bit for bit.
template <class T, int BX_, int BY_, int BZ, int MODE, int ARITH, bool ISO, bool OCT = false, bool MAIL = true>
__global__ void __launch_bounds__(T3GeoOf<T, BX_, BY_, BZ, ARITH>::NT,
                                  (sizeof(T) == 4 || ARITH == ARITH_PAIR) ? T3GeoOf<T, BX_, BY_, BZ, ARITH>::CTAS : 2)
    t3_sweep_kernel(const __grid_constant__ CUtensorMap tm_u, const __grid_constant__ SweepArgs a) {
  using G = T3GeoOf<T, BX_, BY_, BZ, ARITH>;
  using PlaneBits = typename G::PlaneBits;
  constexpr int BX = G::BX, BY = G::BY, W = G::W, PL = G::PL, NZB = G::NZB;
  extern __shared__ __align__(1024) unsigned char sm[];
  T *box = reinterpret_cast<T *>(sm);
  uint32_t *smask = reinterpret_cast<uint32_t *>(sm + G::OFF_MASK);  // [BZ][BY] frozen words of the brick
  PlaneBits *schgp = reinterpret_cast<PlaneBits *>(sm + G::OFF_CHG);  // [BY][BX] planes changed (grid order)
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm + G::OFF_BAR), *grp = bar + 1;
  __shared__ T3Desc s_desc[2];
  __shared__ unsigned long long s_max[OCT ? 8 : 1];  // per sweep: the CTA's change word
  __shared__ unsigned s_chg[OCT ? 1 : G::NB];        // block-change output: the brick's blocks
  __shared__ volatile int s_abort;

  if ((saddr(sm) & 127u) != 0) {  // TMA destinations must be 128-byte aligned
    if (threadIdx.x == 0) {
      atomicCAS(a.err, 0, DEV_ERR_SMEM_ALIGN);
      atomicExch(a.err + 1, 1);
    }
    return;
  }
  const int tid = threadIdx.x, lane = tid & 31;
  const bool compute = tid < G::NC;
  // a block-masked sweep takes tickets only for the bricks with an active block
  const int ntile = a.nticket ? *a.nticket : a.ntx * a.nty * a.ntz;
  const bool masked = a.fmask != nullptr;
  T *__restrict__ u = reinterpret_cast<T *>(a.u);
  const T *__restrict__ capg = reinterpret_cast<const T *>(a.cap);

  if (tid == 0) {
    s_abort = 0;
    mbar_init(bar, 1);
    for (int g = 0; g < G::NG; ++g) mbar_init(grp + g, 1);
    mbar_fence_init();
  }
  // FP64 reference and fast arithmetic: the spacings' constants by sorted order
  constexpr bool kGod64 = kGod64Of<T, ARITH>;
  __shared__ GodPerm64 s_perm[kGod64 ? 6 : 1];
  if (kGod64 && a.kperm) {
    for (int q = tid; q < (int)(6 * sizeof(GodPerm64) / 8); q += G::NT)
      reinterpret_cast<double *>(s_perm)[q] = reinterpret_cast<const double *>(a.kperm)[q];
  }
  __shared__ uint8_t s_col[G::NC];  // diagonal order -> ly * BX + lx
  if (compute) s_col[diag_rank<BX, BY>(tid % BX, tid / BX)] = (uint8_t)tid;
  if (tid < (OCT ? 8 : 1)) s_max[tid] = 0;
  if (!OCT && tid < G::NB) s_chg[tid] = 0;
  __syncthreads();
  int wait_flag = -1, wait_epoch = 0;  // helper warp: an earlier sweep's flag to wait for
  if (!compute) t3_next<G, OCT, MAIL>(a, ntile, s_desc[0], &s_abort, wait_flag, wait_epoch);
  __syncthreads();

  // my column, brick-local x, y in sweep order, by diagonal
  const int col = compute ? s_col[tid] : 0, lx = col % BX, ly = col / BX, lxy = lx + ly;
  for (int it = 0;; ++it) {
    const T3Desc &d = s_desc[it & 1];
    if (d.stop) break;
    const int sxd = d.sx, syd = d.sy, szd = d.sz;
    const int bi = sxd > 0 ? d.li : a.ntx - 1 - d.li;
    const int bj = syd > 0 ? d.lj : a.nty - 1 - d.lj;
    const int bk = szd > 0 ? d.lk : a.ntz - 1 - d.lk;
    const int tile = d.tile;
    const int x0 = 1 + bi * BX, y0 = 1 + bj * BY, z0 = 1 + bk * BZ;
    const int zcnt = min(BZ, a.nz - z0 + 1);  // planes of the brick inside the grid
    // the box: TMA from (x0 - 1, y0 - 1, z0 - 1); out-of-range rows and planes
    // read 0 (never used).  The barrier before orders this CTA's generic accesses
    // to the box (each thread's proxy fence) before the copy's writes; the global
    // fence orders the flags acquired by this warp before the copy's reads.
    if constexpr (OCT || !MAIL) {
      if (!compute) t3_wait(a, wait_flag, wait_epoch, &s_abort);
    }
    if (tid == G::NC) {
      if constexpr (OCT || !MAIL) fence_proxy_async_global();
      mbar_arrive_tx(bar, G::BOX_BYTES);
      tma_load_3d(box, &tm_u, bi * BX, y0 - 1, z0 - 1, bar);
    }
    // frozen words of the brick's rows: node bit (x0 - 1 + gx) & 31
    const int mshift = (bi * BX) & 31;
    bool frozen = false;  // does one of them freeze a node of the brick?
    if (masked) {
      for (int q = tid; q < BZ * BY; q += G::NT) {
        const int p = q / BY, r = q % BY;
        uint32_t w = 0;
        if (p < zcnt && y0 + r <= a.ny)
          w = __ldg(a.fmask + (long long)(z0 + p) * (a.mask_fy * a.mask_fw) +
                    (long long)((bi * BX) >> 5) * a.mask_fy + (y0 - 1 + r));
        smask[q] = w;
        frozen = frozen || ((w >> mshift) & ((1u << BX) - 1u)) != 0;
      }
    }
    const int gxl = sxd > 0 ? lx : BX - 1 - lx;  // my column in grid order
    const int gyl = syd > 0 ? ly : BY - 1 - ly;
    const bool vxy = compute && (x0 + gxl <= a.nx) && (y0 + gyl <= a.ny);
    // replace-update: the cap bounds of my column's 8^3 blocks in this brick
    using CB = CapBound<T, ARITH>;
    typename CB::type bnds[NZB];
#pragma unroll
    for (int q = 0; q < NZB; ++q) {
      bnds[q] = 0;
      if (MODE == MODE_REPLACE && vxy)
        bnds[q] = bk * NZB + q >= a.nbz ? typename CB::type(INFINITY) : CB::load(a, ((long long)(bk * NZB + q) * a.nby + ((y0 - 1 + gyl) >> 3)) * a.nbx + ((x0 - 1 + gxl) >> 3));
    }
    // the box copy has landed (the helper's wait is bounded; on abort it lets it
    // land all the same): the others wait for the helper at the barrier
    if (!compute && !mbar_wait(bar, it & 1, a, tile, &s_abort)) {
      const long long t0 = cycles();
      while (!mbar_try(bar, it & 1) && cycles() - t0 < 4000000000ll) {
      }
    }
    frozen = __syncthreads_or(frozen) != 0;
    mbar_try(bar, it & 1);  // complete: each thread's own view of the copy's writes
    const bool poisoned = tile == a.poison_col;  // test hook: the brick hands nothing over
    const bool mute = !MAIL || poisoned;
    if (!compute) {
      t3_receive<T, G>(a, d, tile, d.epoch, box, x0, y0, zcnt, grp, &s_abort);
      t3_next<G, OCT, MAIL>(a, ntile, s_desc[(it + 1) & 1], &s_abort, wait_flag, wait_epoch);
    } else {
      // the planes of my column that update, one bit each in sweep order (inside
      // the grid, in a visited block, not frozen).  Read once per brick, off the
      // levels' dependency chain; most bricks freeze no node.
      PlaneBits live = 0, changed = 0;
      if (vxy) {
        const unsigned mine = d.act >> ((gyl >> 3) * G::NBX + (gxl >> 3));
#pragma unroll
        for (int q = 0; q < NZB; ++q)
          if ((mine >> (q * G::NBX * G::NBY)) & 1u) live |= PlaneBits(0xff) << (8 * q);
        if (zcnt < BZ) live &= (PlaneBits(1) << zcnt) - 1;
        if (frozen) {
#pragma unroll 8
          for (int p = 0; p < BZ; ++p) live &= ~(PlaneBits((smask[p * BY + gyl] >> (mshift + gxl)) & 1u) << p);
        }
        if (szd < 0) live = G::flip(live);
      }
      // replace-update: the smallest cap bound of my column in this brick
      typename CB::type bnd = bnds[0];
#pragma unroll
      for (int q = 1; q < NZB; ++q) bnd = CB::lower(bnd, bnds[q]);
      // downwind faces: the planes whose x or y face node I send (every node of the
      // face inside the grid: a reader takes those of visited blocks)
      const bool mx = lx == BX - 1 && d.li < a.ntx - 1, my = ly == BY - 1 && d.lj < a.nty - 1;
      PlaneBits face = 0;
      if (vxy && !mute && (mx || my)) {
        face = zcnt < BZ ? (PlaneBits(1) << zcnt) - 1 : PlaneBits(~0ull >> (64 - BZ));
        if (szd < 0) face = G::flip(face);
      }
      // my z face node, the column's last: its level, where a brick is downwind
      const int zlev = vxy && !mute && d.lk < a.ntz - 1 ? lxy + BZ - 1 : -G::GL;
      // mailbox entry of my face node of level L: row L - foff (the reader's level, wrapped)
      const int foff = mx ? BX - 1 : BY - 1, fcol = mx ? G::MX + ly : G::MY + lx;
      // the levels: node (lx, ly, lz = L - lx - ly), sweep order; live, face and
      // changed planes as bits of 32-level words, bit L for the node of level L
      const int dzo = szd > 0 ? PL : -PL;
      T *p = box + (1 + gyl) * W + 1 + gxl + (szd > 0 ? PL : BZ * PL) + (d.lev0 - lxy) * dzo;  // my node of level L
      T tmax = T(0);
      const bool rec = !OCT && a.blk_chg != nullptr;
      float acc = 0.0f;  // block-change output: my change in block accq of my column
      int accq = 0;
      const int accb = (gyl >> 3) * G::NBX + (gxl >> 3);
      const int lev1 = d.lev1;
      auto levels = [&](auto ftz) {
#pragma unroll 1
        for (int L = d.lev0; L < lev1;) {  // lev0 is a multiple of 8
          const int c0 = L & ~31, cend = min(lev1, c0 + 32);
          unsigned m = G::level_word(live, c0 - lxy) >> (L - c0), fm = G::level_word(face, c0 - lxy) >> (L - c0);
          unsigned chgw = 0;
#pragma unroll 1
          for (; L < cend; L += G::GL, m >>= G::GL, fm >>= G::GL) {
            // the faces of the next GL levels (the helper's waits are bounded, and end in an arrival)
            if (tid < 32) {
              while (!mbar_try(grp + L / G::GL, it & 1)) {
              }
            }
            unsigned cg = 0;
#pragma unroll
            for (int i = 0; i < G::GL; ++i, p += dzo) {
              level_bar<G::NC>();
              const unsigned bit = 1u << i;
              if (m & bit) {
                const T v = *p;
                T g;
                if constexpr (kGod64) {
                  g = god64_node<ARITH>(p[-1], p[1], p[-W], p[W], p[-PL], p[PL], a.k64, a.kperm ? s_perm : nullptr);
                } else {
                  // the reference's minima keep grid orientation: min(u[x-1], u[x+1])
                  const T m0 = vmin<T, ARITH>(p[-1], p[1]);
                  const T m1 = vmin<T, ARITH>(p[-W], p[W]);
                  const T m2 = vmin<T, ARITH>(p[-PL], p[PL]);
                  g = local_update<T, MODE, ARITH, ISO, decltype(ftz)::value>(m0, m1, m2, a.k64, a.k32);
                }
                T nv;
                if constexpr (MODE == MODE_REPLACE) {
                  nv = g;
                  if (!(kGod64 ? d_below(g, bnd) : CB::below(g, bnd))) {
                    const int lz = L + i - lxy, gz = szd > 0 ? lz : BZ - 1 - lz;
                    nv = vmin<T, ARITH>(cap_value<T, ARITH>(capg + (long long)(z0 + gz) * a.plane +
                                                            (long long)(y0 + gyl) * a.px + (x0 + gxl)),
                                        g);
                  }
                } else {
                  nv = kGod64 ? d_min(v, g) : vmin<T, ARITH>(v, g);
                }
                if (kGod64 ? d_differ(nv, v) : vdiffers<T, ARITH>(nv, v)) {
                  *p = nv;
                  cg |= bit;
                  T dv = T(0);
                  if (rec || change_may_exceed<T, ARITH>(v, nv, a.hmin, tmax)) {
                    dv = node_change<T, ARITH>(v, nv, a.hmin);
                    tmax = kGod64 ? d_max(tmax, dv) : vmax_nonneg<T, ARITH>(tmax, dv);
                  }
                  if (rec) {
                    const int lz = L + i - lxy, q = (szd > 0 ? lz : BZ - 1 - lz) >> 3;
                    if (q != accq) {
                      if (acc > 0.0f) atomicMax(&s_chg[accq * (G::NBX * G::NBY) + accb], __float_as_uint(acc));
                      accq = q;
                      acc = 0.0f;
                    }
                    acc = fmaxf(acc, change_f<T, ARITH>(dv));
                  }
                }
              }
            }
            if ((unsigned)(zlev - L) < (unsigned)G::GL)
              mail_put<T>(d.mail + (G::MZ + (lxy % BY) * BX + lx) * G::WV, p[(zlev - L - G::GL) * dzo], d.epoch);
            if (fm & ((1u << G::GL) - 1u)) {  // the group's face nodes: the readers take them by groups too
#pragma unroll
              for (int i = 0; i < G::GL; ++i) {
                if ((fm >> i) & 1u) {
                  const T v = p[(i - G::GL) * dzo];
                  int r = L + i - foff;
                  if (r >= BZ) r -= BZ;
                  mail_put<T>(d.mail + (r * (BX == BY || mx ? BY : BX) + fcol) * G::WV, v, d.epoch);
                  if (mx && my) {  // the corner column: its y face too
                    r = L + i - (BY - 1);
                    if (r >= BZ) r -= BZ;
                    mail_put<T>(d.mail + (G::MY + r * BX + lx) * G::WV, v, d.epoch);
                  }
                }
              }
            }
            chgw |= cg << (L - c0);
          }
          changed |= G::plane_bits(chgw, c0 - lxy);
        }
      };
      // the FP32 parts' roots flush subnormals unless the spacings can make one
      constexpr bool kRoots32 = sizeof(T) == 4 || ARITH == ARITH_MIXED || ARITH == ARITH_PAIR;
      if (!kRoots32 || a.k32.tiny)
        levels(std::false_type{});
      else
        levels(std::true_type{});
      if (szd < 0) changed = G::flip(changed);
      schgp[gyl * BX + gxl] = changed;
      if (rec && acc > 0.0f) atomicMax(&s_chg[accq * (G::NBX * G::NBY) + accb], __float_as_uint(acc));
      // the sweep's change word, per CTA
#pragma unroll
      for (int off = 16; off > 0; off >>= 1)
        tmax = vmax_nonneg<T, ARITH>(tmax, __shfl_xor_sync(0xffffffffu, tmax, off));
      if (lane == 0 && change_pos<T, ARITH>(tmax)) {
        unsigned long long w;
        if constexpr (sizeof(T) == 4)
          w = __float_as_uint(tmax);
        else
          w = change_u64<T, ARITH>(tmax);
        atomicMax(&s_max[OCT ? d.sweep : 0], w);
      }
    }
    __syncthreads();  // the box holds the brick's new values
    if (compute) {
      // the rows with a changed node -> global memory, 32 / BX rows a warp
      const int gx = tid % BX, gy = tid / BX;
      PlaneBits row = schgp[tid], any;
#pragma unroll
      for (int off = 1; off < BX; off <<= 1) row |= __shfl_xor_sync(0xffffffffu, row, off);
      any = row;
#pragma unroll
      for (int off = BX; off < 32; off <<= 1) any |= __shfl_xor_sync(0xffffffffu, any, off);
      if (x0 + gx > a.nx || y0 + gy > a.ny) row = 0;
      T *up = u + (long long)z0 * a.plane + (long long)(y0 + gy) * a.px + (x0 + gx);
      const T *bp = box + PL + (1 + gy) * W + 1 + gx;
      const long long pl = a.plane;
#pragma unroll 1
      for (int p = 0; any != 0; p += 4, any >>= 4, row >>= 4, bp += 4 * PL, up += 4 * pl) {
        if ((any & 15u) == 0) continue;
        T v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (row & (1u << i)) v[i] = bp[i * PL];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (row & (1u << i)) up[i * pl] = v[i];
      }
    }
    fence_proxy_async();  // my accesses to the box come before the next copy's writes
    if (__syncthreads_or(s_abort)) break;
    // the brick is done: publish (a round's later sweeps, if any, wait for it, and
    // without mail the downwind bricks).  The barrier orders every thread's stores
    // before this thread's GPU-scope fence, which orders them before the flag.
    if constexpr (OCT || !MAIL) {
      if (tid == G::NC && !poisoned && a.tflag) publish_gpu(a.tflag + tile, d.epoch);
    }
    if (!OCT && a.blk_chg != nullptr && tid < G::NB) {
      // block changes: only nodes inside the grid change, so a positive one names a block of the grid
      if (s_chg[tid]) {
        const int bx = G::NBX * bi + tid % G::NBX, by = G::NBY * bj + (tid / G::NBX) % G::NBY;
        const int bz = NZB * bk + tid / (G::NBX * G::NBY);
        a.blk_chg[((long long)bz * a.nby + by) * a.nbx + bx] = s_chg[tid];
        s_chg[tid] = 0;
      }
    }
  }
  // the CTA's change words -> the sweeps' counters
  __syncthreads();
  if (tid < (OCT ? 8 : 1) && s_max[tid]) {
    if constexpr (OCT) {  // FP32: the low word of the sweep's 64-bit slot
      atomicMax(reinterpret_cast<unsigned long long *>(a.maxchg) + tid, s_max[tid]);
    } else if constexpr (sizeof(T) == 4) {
      atomicMax(reinterpret_cast<unsigned int *>(a.maxchg), (unsigned)s_max[0]);
    } else {
      atomicMax(reinterpret_cast<unsigned long long *>(a.maxchg), s_max[0]);
    }
  }
}

}  // namespace pdfs
