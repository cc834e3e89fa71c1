// Candidates extended exactly (included by hz_wave.cuh after hz_gate2.cuh).
//
// The lockstep gate hands on every hit whose extensions may reach the
// threshold, and those that run past its cell cap (src/gpu/kernels.rs:1279-1406
// extends every hit warp-wide).  long_kernel extends each candidate of a wave
// to its end over the 2-bit packed sequences and finds in each direction the
// maximum and the first cell that reaches it.  It writes them into the
// candidate and marks it kDoneFlag, so the exact kernel is left with the
// entropy and the accept.
//
// Few candidates (LongArgs::wide_max; all of them where costs are kWide, whose
// group states would not fit 16 bits) go half a warp per direction, 256 cells
// per step (long_wide): their time is that of the longest extension.  More go
// one lane per candidate-direction, in rounds of kRound cells, which takes
// fewer instructions per cell.  There the maximum's position is found without
// a per-cell test: in a round whose cells are all valid the main pass notes
// the last eight-cell group in which the running maximum rose (the first cell
// reaching the round's final maximum lies in it) together with that group's
// starting sum, and only when the direction ends is that one group rescored.
// A round that stops early (a drop, a special base, the edge) searches its own
// valid groups at once, from the group states it keeps in shared memory and
// the codes it still holds in registers.  Scores come from the gate's lookup
// (costs by byte permute, sums by dot product): 3.5 M candidates 2.76 ms, with
// a shared-memory lookup per cell 3.13.
//
// Semantics are exact_dir4's: cells counted up to and including the first
// dropping cell (or to the edge); the right position is the cell offset of
// the maximum (-1 when the maximum is the empty extension's 0), the left one
// the offset + 1 (0 then).
#pragma once

namespace hz {

constexpr int kRound = 48;             // cells long_kernel scores per round
constexpr int kChunks = kRound / 16;   // 16-cell code words per sequence in a round
constexpr int kGroups = kRound / 8;    // eight-cell groups per round

// The kRound bases of a packed half that start at base p: their codes, 16
// per word, and their special bits (cells 0..31 in *sp_lo, the rest in
// *sp_hi), from the 16-byte records that hold them.
__device__ __forceinline__ void window_round(const uint4 *__restrict__ blk, uint32_t p, uint32_t code[kChunks],
                                             uint32_t *sp_lo, uint32_t *sp_hi) {
  constexpr int kRec = (kRound + 31) / 32 + 1;
  uint4 r[kRec];
#pragma unroll
  for (int i = 0; i < kRec; i++) r[i] = __ldg(blk + (p >> 5) + i);
  uint32_t c[2 * kRec];
#pragma unroll
  for (int i = 0; i < kRec; i++) {
    c[2 * i] = r[i].x;
    c[2 * i + 1] = r[i].y;
  }
  const uint32_t o = p & 31u, sh = (o & 15u) << 1;
  const bool upper = o >= 16;  // the window starts in a record's second code word
  uint32_t cs[kChunks + 1];
#pragma unroll
  for (int k = 0; k <= kChunks; k++) cs[k] = upper ? c[k + 1] : c[k];
#pragma unroll
  for (int k = 0; k < kChunks; k++) code[k] = __funnelshift_r(cs[k], cs[k + 1], sh);
  *sp_lo = __funnelshift_r(r[0].z, r[1].z, o);
  *sp_hi = kRound > 32 ? __funnelshift_r(r[1].z, r[kRec - 1].z, o) : 0u;
}

// The costs (negated scores) of the eight cells whose codes are the low 16 bits
// of r and q; and s plus the score of cell k of them.
template <int MODE>
__device__ __forceinline__ Cells8<MODE> costs8(const CostTable<MODE> &tab, uint32_t r, uint32_t q) {
  const uint2 sel = CostTable<MODE>::index(r, q);
  return tab.cells(sel.x, sel.y);
}
template <int MODE> __device__ __forceinline__ int32_t add_score(int32_t s, const Cells8<MODE> &c, int k) {
  static_assert(MODE != kWide, "the lane rounds' sums");
  return __dp4a((int)cost_word(c, k), (int)((MODE == kGeneral ? 1u : 0xFFu) << (8 * (k >> 1))), s);
}

__device__ __forceinline__ int32_t wadd(int32_t a, int32_t b) { return (int32_t)((uint32_t)a + (uint32_t)b); }

// The value v with v = h (mod 2^16) and base - 32768 <= v < base + 32768.
// A round's group states are read back against the running sum after all
// its kRound cells, which lies within kRound * 128 of every stored sum; a
// stored maximum read back exceeds its sum by at most xdrop plus one group's
// fall, so every value read lies within kRound * 255 + xdrop of the base
// (cost_mode in hz_engine.cu admits only matrices and xdrops that keep this below 32768).
__device__ __forceinline__ int32_t near16(int32_t base, uint32_t h) {
  return wadd(base, (int32_t)(int16_t)(uint16_t)(h - (uint32_t)base));
}

constexpr uint32_t kDoneFlag = 1u << 30;  // Cand::call: maxima and positions filled in by long_kernel

struct LongArgs {
  const uint4 *ref, *refr, *qry, *qryr;  // packed halves (pack2_kernel)
  const uint8_t *ref8, *qry8;            // 8-bit codes of the target and of the query store
  uint32_t rlen, qtotal;
  const CallDev *calls;
  Cand *cand;
  uint32_t cand_cap;
  WaveTotals *tot;
  int32_t sub[64];
  int32_t xdrop;
  uint32_t late_max_safe;  // as GateArgs::late_max_safe
  uint32_t wide_max;       // candidates up to which half a warp extends each direction (kWide: always)
};

struct LongWarp {
  uint32_t queue[64];          // long candidates claimed by the warp, not yet on a lane
  uint32_t grp[kGroups][32];   // the sum (low half) and maximum (high half) before each group of a round
};

struct LongSmem {
  LongWarp warp[kGateWarps];
};

// The first of the eight cells whose codes are the low 16 bits of r and q at
// which the running sum, starting from s, equals target (8 if none does).
template <int MODE>
__device__ __forceinline__ uint32_t first_reach(const CostTable<MODE> &tab, uint32_t r, uint32_t q, int32_t s, int32_t target) {
  const Cells8<MODE> cost = costs8(tab, r, q);
  uint32_t c = 8;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    s = add_score(s, cost, i);
    if (c == 8 && s == target) c = (uint32_t)i;
  }
  return c;
}

// Few candidates: half a warp per direction, sixteen cells per lane, 256 per
// step.  A wave's time here is that of its longest extension, and lanes on
// their own need a 48-cell round for what a step does for 256 cells.  A lane
// sums its cells' costs A (negated scores), and notes their minimum, maximum
// and largest rise over an earlier minimum; scans over the half warp give the
// cost and the minimum before its cells, and with them whether one of its
// cells drops.  The first lane that has one finds which; the minimum's first
// cell is looked for where a step lowers it.
template <int MODE> __device__ __forceinline__ void long_wide(const LongArgs &a, uint32_t ncand) {
  const uint32_t lane = threadIdx.x & 31, l = lane & 15u, half = lane >> 4;  // half 0: right, 1: left
  const CostTable<MODE> tab(a.sub);
  const int32_t X = a.xdrop;
  const uint4 *const rseq = half ? a.refr : a.ref, *const qseq = half ? a.qryr : a.qry;
  unsigned long long cells_acc = 0;
  uint32_t i = 0;
  if (lane == 0) i = atomicAdd(&a.tot->long_next, 1u);
  i = __shfl_sync(0xffffffffu, i, 0);
  while (i < ncand) {
    uint32_t next = 0;  // claimed while this one is extended
    if (lane == 0) next = atomicAdd(&a.tot->long_next, 1u);
    const Cand c = a.cand[i];
    const CallDev cd = a.calls[c.call & ~(kLongFlag | kDoneFlag)];
    const uint32_t edge = !(c.call & kLongFlag) ? 0u
                          : half                ? min(c.r0, c.q0 - cd.qoff)
                                                : min(a.rlen - c.r0, cd.qoff + cd.qlen - c.q0);
    const uint32_t rp = half ? a.rlen - c.r0 : c.r0, qp = half ? a.qtotal - c.q0 : c.q0;
    // the half's state: cost and minimum at the step's start, the minimum's
    // cell (-1: none yet), cells scored
    int32_t at = 0, low = 0, pos = -1;
    uint32_t cells = 0;
    bool done = edge == 0;
    for (uint32_t step = 0; __any_sync(0xffffffffu, !done); step += 256) {
      const uint32_t k0 = step + 16 * l;
      const uint32_t v = done || k0 >= edge ? 0u : min(edge - k0, 16u);  // the lane's cells
      uint32_t rlo, rhi, rsp, qlo, qhi, qsp;
      window32(rseq, v ? rp + k0 : 0u, &rlo, &rhi, &rsp);
      window32(qseq, v ? qp + k0 : 0u, &qlo, &qhi, &qsp);
      const uint2 sel = CostTable<MODE>::index(rlo, qlo);
      const Cells8<MODE> c8[2] = {tab.cells(sel.x, sel.y), tab.cells(sel.x >> 16, sel.y >> 16)};
      int32_t A[16];
#pragma unroll
      for (int j = 0; j < 16; j++) {
        const int32_t cost = (int32_t)add_cost(c8[j >> 3], j & 7, 0u);
        A[j] = (uint32_t)j < v ? cost : 0;
      }
      uint32_t sp = (rsp | qsp) & ((1u << v) - 1u);
      if (__any_sync(0xffffffffu, sp != 0)) {  // special bases: their scores from the 8-bit codes
#pragma unroll
        for (int j = 0; j < 16; j++)
          if (sp >> j & 1u) {
            const uint32_t pr = rp + k0 + j, pq = qp + k0 + j;
            A[j] = -a.sub[a.ref8[half ? a.rlen - 1u - pr : pr] * kNuc + a.qry8[half ? a.qtotal - 1u - pq : pq]];
          }
      }
      int32_t lm = 0x7FFFFFFF, hi = -0x7FFFFFFF, rise = 0;
#pragma unroll
      for (int j = 0; j < 16; j++) {
        if (j) A[j] = wadd(A[j], A[j - 1]);
        lm = min(lm, A[j]);
        hi = max(hi, A[j]);
        rise = max(rise, A[j] - lm);
      }
      if (v == 0) lm = 0x3FFFFFFF;  // no cells: never the minimum, never a drop
      int32_t incl = A[15];
#pragma unroll
      for (int d = 1; d < 16; d <<= 1) {
        const int32_t up = __shfl_up_sync(0xffffffffu, incl, d, 16);
        if (l >= (uint32_t)d) incl = wadd(incl, up);
      }
      const int32_t mine = wadd(at, incl - A[15]);  // the cost before the lane's cells
      int32_t upto = v ? wadd(mine, lm) : 0x7FFFFFFF;
#pragma unroll
      for (int d = 1; d < 16; d <<= 1) upto = min(upto, __shfl_up_sync(0xffffffffu, upto, d, 16));
      int32_t before = __shfl_up_sync(0xffffffffu, upto, 1, 16);
      before = l ? min(before, low) : low;  // the minimum before them
      const int32_t D = mine - before;
      const bool drops = v && (hi > X - D || rise > X);
      const uint32_t fl = __ballot_sync(0xffffffffu, drops) >> (16 * half) & 0xFFFFu;
      const uint32_t f = fl ? (uint32_t)(__ffs((int)fl) - 1) : 16u;  // the first lane with a drop
      // the cells before the drop: their number, and the lowest cost
      uint32_t n = l < f ? v : 0u;
      if (l == f) {
        int32_t m = -D, best = 0x3FFFFFFF;
        uint32_t hit = 16;
#pragma unroll
        for (int j = 0; j < 16; j++) {
          m = min(m, A[j]);
          if (hit == 16) {
            if (A[j] - m > X && (uint32_t)j < v) hit = (uint32_t)j;
            else best = min(best, A[j]);
          }
        }
        n = hit;
        lm = best;
      }
      const int32_t least = n ? wadd(mine, lm) : 0x7FFFFFFF;
      int32_t all = least;
#pragma unroll
      for (int d = 1; d < 16; d <<= 1) all = min(all, __shfl_xor_sync(0xffffffffu, all, d));
      if (__any_sync(0xffffffffu, !done && all < low)) {  // a new minimum: its first cell
        uint32_t first = 16;
#pragma unroll
        for (int j = 15; j >= 0; j--)
          if ((uint32_t)j < n && wadd(mine, A[j]) == all) first = (uint32_t)j;
        const uint32_t has = __ballot_sync(0xffffffffu, first < 16) >> (16 * half) & 0xFFFFu;
        const uint32_t g = has ? (uint32_t)(__ffs((int)has) - 1) : 0u;
        const uint32_t cell = step + 16 * g + __shfl_sync(0xffffffffu, first, g, 16);
        if (!done && all < low) {
          low = all;
          pos = (int32_t)cell;
        }
      }
      const uint32_t in_f = __shfl_sync(0xffffffffu, n, f & 15u, 16);
      at = wadd(at, __shfl_sync(0xffffffffu, incl, 15, 16));
      if (!done) {
        if (f < 16) {
          cells = step + 16 * f + in_f + 1;
          done = true;
        } else if (step + 256 >= edge) {
          cells = edge;
          done = true;
        }
      }
    }
    const int32_t lmax = __shfl_sync(0xffffffffu, -low, 16), lpos = __shfl_sync(0xffffffffu, pos, 16);
    const uint32_t lcells = __shfl_sync(0xffffffffu, cells, 16);
    if (lane == 0 && (c.call & kLongFlag)) {
      Cand &out = a.cand[i];
      out.rmax = -low;
      out.lmax = lmax;
      out.rpos = pos;
      out.lpos = lpos + 1;
      out.call = c.call | kDoneFlag;
      cells_acc += cells + lcells;
    }
    i = __shfl_sync(0xffffffffu, next, 0);
  }
  if (lane == 0 && cells_acc) atomicAdd(&a.tot->cells, cells_acc);
}

// More candidates: a lane per candidate and direction, in rounds of kRound cells.
template <int MODE> __device__ __forceinline__ void long_lanes(const LongArgs &a, uint32_t ncand) {
  static_assert(MODE != kWide, "group states are kept modulo 2^16 (near16)");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  LongSmem &sm = *reinterpret_cast<LongSmem *>(smem_raw);
  LongWarp &wp = sm.warp[threadIdx.x >> 5];
  const CostTable<MODE> tab(a.sub);
  const uint32_t lane = threadIdx.x & 31;
  const int32_t X = a.xdrop;
  unsigned long long cells_acc = 0;
  uint32_t qn = 0;  // candidates in the warp's queue (warp-uniform)
  bool exhausted = false;

  // lane state: the candidate (index, anchors, left edge, call word), the
  // direction, the next round's first base in the direction's packed halves,
  // cells left to the edge, running sum and maximum, cells scored in the
  // direction and in both, the maximum's first cell (-1: none yet) or the
  // group that holds it (pbase >= 0, with the group's starting sum pS), and
  // the right direction's result
  bool have = false;
  uint32_t ci = 0, r0 = 0, q0 = 0, nl = 0, dir = 0, rp = 0, qp = 0, n = 0, cells = 0, tcells = 0;
  int32_t S = 0, M = 0, mpos = -1, pbase = -1, pS = 0, rmax = 0, rpos = -1;
  auto start = [&](uint32_t d, uint32_t edge) {
    dir = d;
    n = edge;
    rp = d ? a.rlen - r0 : r0;
    qp = d ? a.qtotal - q0 : q0;
    S = 0;
    M = 0;
    cells = 0;
    mpos = -1;
    pbase = -1;
  };
  while (true) {
    const unsigned need = __ballot_sync(0xffffffffu, !have);
    if (need && qn < (uint32_t)__popc(need) && !exhausted) {
      // claim chunks of 32 candidates and queue the long ones
      while (qn < 32 && !exhausted) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&a.tot->long_next, 32u);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= ncand) {
          exhausted = true;
          break;
        }
        const uint32_t idx = base + lane;
        const bool lg = idx < ncand && (a.cand[idx].call & kLongFlag) != 0;
        const unsigned b = __ballot_sync(0xffffffffu, lg);
        if (lg) wp.queue[qn + (uint32_t)__popc(b & lanemask_lt())] = idx;
        qn += (uint32_t)__popc(b);
      }
      __syncwarp();
    }
    if (need && qn) {
      const uint32_t k = (uint32_t)__popc(need & lanemask_lt());
      if (!have && k < qn) {
        ci = wp.queue[qn - 1 - k];
        const Cand c = a.cand[ci];
        const CallDev cd = a.calls[c.call & ~(kLongFlag | kDoneFlag)];
        r0 = c.r0;
        q0 = c.q0;
        nl = min(r0, q0 - cd.qoff);
        have = true;
        tcells = 0;
        start(0, min(a.rlen - r0, cd.qoff + cd.qlen - q0));
      }
      qn -= min((uint32_t)__popc(need), qn);
      __syncwarp();
    }
    if (!__any_sync(0xffffffffu, have)) {
      if (exhausted && qn == 0) break;
      continue;
    }
    if (!have) n = 0;  // an idle lane scores an empty window at base 0
    const uint32_t prp = have ? rp : 0u, pqp = have ? qp : 0u;
    uint32_t Rc[kChunks], Qc[kChunks], RS0, RS1, QS0, QS1;
    window_round(dir ? a.refr : a.ref, prp, Rc, &RS0, &RS1);
    window_round(dir ? a.qryr : a.qry, pqp, Qc, &QS0, &QS1);
    const uint32_t v = min(n, (uint32_t)kRound);
    const uint32_t sp0 = (RS0 | QS0) & (v >= 32 ? 0xFFFFFFFFu : ((1u << v) - 1u));
    const uint32_t sp1 = (RS1 | QS1) & (v >= 64 ? 0xFFFFFFFFu : v > 32 ? ((1u << (v - 32)) - 1u) : 0u);
    const uint32_t vv = sp0 ? (uint32_t)(__ffs(sp0) - 1) : sp1 ? 32u + (uint32_t)(__ffs(sp1) - 1) : v;

    // the gate's main pass, noting the last group in which the maximum rose
    uint32_t flags = 0;
    int32_t gi = -1;
#pragma unroll
    for (int h = 0; h < kChunks; h++) {
      const uint2 sel = CostTable<MODE>::index(Rc[h], Qc[h]);
#pragma unroll
      for (int gg = 0; gg < 2; gg++) {
        const int g = 2 * h + gg;
        wp.grp[g][lane] = __byte_perm((uint32_t)S, (uint32_t)M, 0x5410u);
        const int32_t Mg = M;
        const Cells8<MODE> cost = tab.cells(gg ? sel.x >> 16 : sel.x, gg ? sel.y >> 16 : sel.y);
        int32_t lo = 0x7FFFFFFF;
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          const int32_t S1 = add_score(S, cost, i);
          const int32_t S2 = add_score(S1, cost, i + 1);
          M = __vimax3_s32(M, S1, S2);
          lo = __vimin3_s32(lo, S1, S2);
          S = S2;
        }
        flags |= (uint32_t)((int32_t)((uint32_t)M - (uint32_t)lo) > X) << g;
        gi = M > Mg ? g : gi;
      }
    }
    // the exact end of the round: the flagged groups in turn, cell by cell
    const uint32_t gv = vv >> 3;
    uint32_t todo = have ? (flags | (gv < (uint32_t)kGroups ? 1u << gv : 0u)) & ((2u << gv) - 1u) : 0u;
    bool ended = false, dropped = false;
    int32_t res = 0;
    uint32_t used = kRound;
    int32_t Sf = S, Mf = M;
    while (__any_sync(0xffffffffu, todo != 0)) {
      if (todo) {
        const uint32_t g = (uint32_t)(__ffs(todo) - 1);
        todo &= todo - 1;
        const uint32_t st = wp.grp[g][lane];
        int32_t Se = near16(S, st & 0xFFFFu), Me = near16(S, st >> 16);
        const uint32_t ch = g >> 1;
        uint32_t hw = Rc[0], qw = Qc[0];
#pragma unroll
        for (int k = 1; k < kChunks; k++)
          if (ch == (uint32_t)k) {
            hw = Rc[k];
            qw = Qc[k];
          }
        const uint32_t sh = (g & 1u) << 4;
        const Cells8<MODE> cost = costs8(tab, hw >> sh, qw >> sh);
        if (a.late_max_safe && g != gv) {
          int32_t D = (int32_t)((uint32_t)Me - (uint32_t)Se);
          uint32_t dm = 0;
#pragma unroll
          for (int i = 0; i < 8; i++) {
            D = max((int32_t)add_cost(cost, i, (uint32_t)D), 0);
            dm |= (uint32_t)(D > X) << i;
          }
          if (dm) {
            ended = dropped = true;
            res = g + 1 < (uint32_t)kGroups ? near16(S, wp.grp[g + 1][lane] >> 16) : M;
            used = 8 * g + (uint32_t)(__ffs(dm) - 1) + 1;
            todo = 0;
          }
          continue;
        }
        const uint32_t lim = g == gv ? vv - 8 * g : 8u;
        uint32_t d = 8;
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const int32_t Sx = add_score(Se, cost, i);
          const int32_t Mx = max(Me, Sx);
          if ((uint32_t)i < lim && d == 8) {
            if ((int32_t)((uint32_t)Mx - (uint32_t)Sx) > X) {
              d = (uint32_t)i;
            } else {
              Se = Sx;
              Me = Mx;
            }
          }
        }
        if (d < 8) {
          ended = dropped = true;
          res = Me;
          used = 8 * g + d + 1;
          todo = 0;
        } else if (g == gv) {
          Sf = Se;
          Mf = Me;
          used = vv;
          todo = 0;
        }
      }
    }
    if (have) {
      bool special_max = false;
      if (!dropped && vv < (uint32_t)kRound && vv < v) {  // a special base at cell vv
        const uint32_t pr = rp + vv, pq = qp + vv;
        const uint32_t r8 = dir ? a.rlen - 1u - pr : pr, q8 = dir ? a.qtotal - 1u - pq : pq;
        const int32_t Sx = wadd(Sf, a.sub[a.ref8[r8] * kNuc + a.qry8[q8]]);
        const int32_t Mx = max(Mf, Sx);
        used = vv + 1;
        if ((int32_t)((uint32_t)Mx - (uint32_t)Sx) > X) {
          ended = dropped = true;
          res = Mf;
        } else {
          special_max = Sx > Mf;
          Sf = Sx;
          Mf = Mx;
        }
      }
      // where the maximum the round ends with was first reached
      const int32_t Mr = dropped ? res : Mf;
      const int32_t M0 = near16(S, wp.grp[0][lane] >> 16);  // the maximum at the round's start
      if (special_max) {
        mpos = (int32_t)(cells + vv);
        pbase = -1;
      } else if (Mr > M0) {
        // every cell valid: the main pass's last rise (a special base at the
        // last cell scores as an A there, which may look like one)
        if (!dropped && vv == (uint32_t)kRound) {
          pbase = (int32_t)(cells + 8u * (uint32_t)gi);
          pS = near16(S, wp.grp[gi][lane] & 0xFFFFu);
        } else {  // the last valid group that starts below Mr holds the first cell reaching it
          uint32_t g = (used - 1) >> 3;
          while (g > 0 && near16(S, wp.grp[g][lane] >> 16) >= Mr) g--;
          static_assert(kChunks == 3, "the chunk select below names three code words");
          const uint32_t hw = (g >> 1) == 0 ? Rc[0] : (g >> 1) == 1 ? Rc[1] : Rc[2];
          const uint32_t qw = (g >> 1) == 0 ? Qc[0] : (g >> 1) == 1 ? Qc[1] : Qc[2];
          const uint32_t sh = (g & 1u) << 4;
          mpos = (int32_t)(cells + 8u * g +
                           first_reach(tab, hw >> sh, qw >> sh, near16(S, wp.grp[g][lane] & 0xFFFFu), Mr));
          pbase = -1;
        }
      }
      if (!dropped) {
        S = Sf;
        M = Mf;
        if (used >= n) {
          ended = true;
          res = M;
        }
      }
      cells += used;
      rp += used;
      qp += used;
      n -= min(used, n);
    }
    if (ended) {
      if (pbase >= 0) {  // rescore the group noted by the main pass
        const uint32_t at = (uint32_t)pbase - cells;  // negative offset from rp, as uint32 arithmetic
        uint32_t rlo, rhi, rsp, qlo, qhi, qsp;
        window32(dir ? a.refr : a.ref, rp + at, &rlo, &rhi, &rsp);
        window32(dir ? a.qryr : a.qry, qp + at, &qlo, &qhi, &qsp);
        mpos = pbase + (int32_t)first_reach(tab, rlo, qlo, pS, res);
        pbase = -1;
      }
      tcells += cells;
      if (dir == 0) {
        rmax = res;
        rpos = mpos;
        start(1, nl);
      } else {
        Cand &c = a.cand[ci];
        c.rmax = rmax;
        c.lmax = res;
        c.rpos = rpos;
        c.lpos = mpos + 1;
        c.call |= kDoneFlag;
        cells_acc += tcells;
        have = false;
      }
    }
  }
  for (int d = 16; d > 0; d >>= 1) cells_acc += __shfl_down_sync(0xffffffffu, cells_acc, d);
  if (lane == 0 && cells_acc) atomicAdd(&a.tot->cells, cells_acc);
}

template <int MODE>
__global__ void __launch_bounds__(kGateThreads) long_kernel(const __grid_constant__ LongArgs a) {
  const uint32_t ncand = min(a.tot->cand, a.cand_cap);
  if constexpr (MODE == kWide) {
    long_wide<MODE>(a, ncand);
  } else {
    if (ncand <= a.wide_max) long_wide<MODE>(a, ncand);
    else long_lanes<MODE>(a, ncand);
  }
}

}  // namespace hz
