// Lockstep score gate over 2-bit packed sequences (included by hz_wave.cuh).
//
// The same work as gate_kernel -- fused hit expansion and the X-drop score
// bound of every hit, src/gpu/kernels.rs:521-1057 -- organised so that a
// warp's 32 lanes run one instruction stream:
//   * a lane owns one hit and scores both of its extensions in one round over
//     one window of each sequence, kLeft bases before the anchor and kRight
//     after it.  Random hits end after ~40 cells to the left (19 of them the
//     seed) and ~21 to the right, so one round ends 92 % of the hits; a lane
//     whose extension goes on keeps its hit for another round, with the
//     anchor moved to where the extension stands;
//   * both extensions read the same forward copy of each sequence: the left
//     one takes its cells in descending order, which costs nothing because
//     every cell's place in the window is a constant of the code;
//   * the sums of the two extensions run as the two 16-bit halves of one
//     word, so one min, max or test serves two cells;
//   * costs are looked up four cells at a time: one byte permute of eight
//     table bytes by four 3-bit indices, and one dot product adds a cell's
//     byte to the running cost;
//   * after a round the lanes rescore the one eight-cell group that holds the
//     first drop of each extension, again both extensions at once, to count
//     the cells up to it.
// Bases that are not uppercase ACGT (soft-masked, N, other, separator) are
// marked in a side mask and end an extension whenever their score alone
// exceeds xdrop, which the engine knows from the matrix.
//
// What bounds it: the integer pipe that runs permutes, shifts, logic and
// min/max at half rate (PRMT, SHF, LOP3 and VIMNMX each measured at one warp
// instruction per two cycles, and together no faster), and the L1 tag stage,
// which takes one cycle per distinct line of a load whatever its width (a
// divergent 16-byte load costs 32 cycles).  Hence sums by IDP and IMAD, which
// run beside that pipe, and one window of four 16-byte records per sequence
// instead of six for two separate ones.
//
// Measured against the kernel before it (one direction per round over two
// packed copies, a shared-memory table lookup and three adds per cell): a 200
// Mbp target took 60.1 ps per hit and takes 36.5 (326.6 -> 198.3 ms for 5.4e9
// hits), a 10 Mbp bin 68 -> 47 ps.
//
// The extension semantics are those of the scalar oracle and the reference
// warp kernel: S += sub[r][q]; M' = max(M, S) includes the cell; the
// extension stops at the first cell with M' - S > xdrop and keeps the maximum
// from before it, or at the edge.  The kernel runs them on A = -S and the
// running minimum of A.  The gate needs the exact cell count of every
// extension, but of the maxima only whether they can sum to hspthresh: it
// bounds each by the maximum over the whole window its extension ends in (a
// superset of the cells that count).  A hit whose bound reaches hspthresh
// ((i32)(f32)total >= hspthresh, monotone in the total) becomes a candidate
// that long_kernel extends exactly; so does one that runs past `cap` cells or
// meets a base that is not ACGT and does not end it by itself.  The exact
// kernel's own test then decides, so the accepted HSPs are the same.
#pragma once

namespace hz {

constexpr int kRight = 40;                    // cells right of the anchor in a round
constexpr int kLeft = 56;                     // cells left of it
constexpr int kWindow = kRight + kLeft;       // bases of a round's window
constexpr int kWinChunks = kWindow / 16;      // 16-base code words of a window
constexpr int kSolo = (kLeft - kRight) / 8;   // the left extension's first groups, scored without a partner
constexpr int kGroupsL = kLeft / 8;           // eight-cell groups of each direction
constexpr int kGroupsR = kRight / 8;
constexpr uint32_t kMaxTile = 256;
// Running costs are kept as kCostBase + A in 16 unsigned bits.  A falls by at
// most kLeft * 127 in a round and rises by at most kLeft * 128 above
// kCostBase + xdrop.
constexpr uint32_t kCostBase = kLeft * 128;
static_assert(kWindow == 96, "a window is read as four 32-base records, at any offset in the first");
static_assert(kLeft % 8 == 0 && kRight % 8 == 0 && kLeft > kRight, "groups of eight cells; the left extension is longer");
// The largest xdrop the 16-bit halves hold: the drop test adds 0x7FFF - xdrop
// to a drawdown and reads bit 15, and the rescoring takes that word down by
// up to 128 per cell.
constexpr int32_t kGate2MaxXdrop = 32767 - 128;

// Shared memory of one warp; slot[] follows with one entry per hit of a tile.
struct GateWarp {
  uint2 sel[kWinChunks][32];    // each lane's table indices: of the even and the odd cells of 16 bases
  uint32_t grp[kGroupsL][32];   // drawdowns before each group, biased (right low half, left high half)
  uint32_t bits[kMaxTile / 32];   // tile hits at which a slot starts
  uint32_t carry[kMaxTile / 32];  // the last slot that starts before the 32 hits
  uint32_t hdr[4];              // the claimed next tile's first position, the position after it, its call
};
// A slot is a run of tile hits of one (position, seed), indexed by its first
// hit: x = pos_table index of tile hit 0 of the run (so hit t is x + t),
// y = query anchor (absolute), z = call, w = cells to the query's right edge |
// cells to its left edge << 16 (each saturated).
inline size_t gate2_smem(int tile) { return kGateWarps * (sizeof(GateWarp) + (size_t)tile * sizeof(uint4)); }

struct Gate2Args {
  GateArgs g;
  // packed forward halves (pack2_kernel's records) from two records before
  // their first base: a window may start kLeft bases before the sequence.
  // Component w of the first record holds the non-ACGT codes of the sequence.
  const uint4 *ref, *qry;
  uint32_t tile;        // hits per warp tile, a multiple of 32, at most kMaxTile
  uint32_t soft_codes;  // bit c: code c (4..7) does not end every extension that meets it
};

// 4-byte global -> shared copy that completes asynchronously (no register
// holds the value), and the wait for all of the thread's copies.
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)),
               "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Byte permute of (a, b); unlike __byte_perm's documented contract, a set top
// bit of a selector nibble replicates the chosen byte's sign.
__device__ __forceinline__ uint32_t permute(uint32_t a, uint32_t b, uint32_t s) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(s));
  return d;
}

// The kWindow bases that start kLeft before base `a` of a packed half: their
// codes, 16 per word, and their special bits, 32 per word.
__device__ __forceinline__ void window_codes(const uint4 r[4], uint32_t a, uint32_t code[kWinChunks],
                                             uint32_t sp[3]) {
  const uint32_t c[8] = {r[0].x, r[0].y, r[1].x, r[1].y, r[2].x, r[2].y, r[3].x, r[3].y};
  const uint32_t o = (a + (64 - kLeft)) & 31u, sh = (o & 15u) << 1;
  const bool upper = o >= 16;  // the window starts in a record's second code word
  uint32_t cs[kWinChunks + 1];
#pragma unroll
  for (int k = 0; k <= kWinChunks; k++) cs[k] = upper ? c[k + 1] : c[k];
#pragma unroll
  for (int k = 0; k < kWinChunks; k++) code[k] = __funnelshift_r(cs[k], cs[k + 1], sh);
#pragma unroll
  for (int k = 0; k < 3; k++) sp[k] = __funnelshift_r(r[k].z, r[k + 1].z, o);
}

// Costs (negated scores) of ACGT pairs as table bytes.  The index of a pair
// is reference ^ query | parity << 2, parity the xor of the reference code's
// two bits: with A C G T = 0..3 a complement flips both bits, so a matrix
// with equal scores for complementary pairs -- HOXD70, and any matrix that
// treats the strands alike -- has one score per index.  GENERAL matrices add
// the reference code's low bit as bit 3 and hold a second table for it.
template <bool GENERAL>
struct CostTable {
  uint32_t t[GENERAL ? 4 : 2];
  __device__ __forceinline__ explicit CostTable(const int32_t *sub) {
#pragma unroll
    for (int i = 0; i < (GENERAL ? 4 : 2); i++) {
      t[i] = 0;
#pragma unroll
      for (int x = 0; x < 4; x++) {
        const int low = i >> 1, parity = i & 1;
        const int r = (parity ^ low) << 1 | low;
        t[i] |= (uint32_t)(uint8_t)(-sub[r * kNuc + (r ^ x)]) << (8 * x);
      }
    }
  }
  // The indices of 16 cells' pairs, a nibble each: even cells, odd cells.
  __device__ __forceinline__ static uint2 index(uint32_t r, uint32_t q) {
    const uint32_t x = r ^ q;
    const uint32_t p = (r ^ (r >> 1)) & 0x55555555u;
    uint2 e;
    e.x = (x & 0x33333333u) | ((p << 2) & ~0x33333333u);
    e.y = ((x >> 2) & 0x33333333u) | (p & ~0x33333333u);
    if (GENERAL) {
      e.x |= (r & 0x11111111u) << 3;
      e.y |= (r << 1) & 0x88888888u;
    }
    return e;
  }
  // The costs of the four cells whose indices are the low nibbles of s.
  __device__ __forceinline__ uint32_t costs(uint32_t s) const {
    if (!GENERAL) return permute(t[0], t[1], s);
    const uint32_t lo = s & 0x7777u;
    // bit 3 of each nibble as a byte mask: nibble 9 takes the sign of byte 1
    const uint32_t m = permute(0x00008000u, 0u, ((s >> 3) & 0x1111u) * 9u);
    return (permute(t[0], t[1], lo) & ~m) | (permute(t[GENERAL ? 2 : 0], t[GENERAL ? 3 : 1], lo) & m);
  }
};

// Cell k (0..7) of an eight-cell group whose costs are e (even bases) and o
// (odd bases): ascending bases for the right extension, descending for the
// left one.  Which word, and which of its bytes.
__device__ __forceinline__ constexpr int right_byte(int k) { return k >> 1; }
__device__ __forceinline__ constexpr int left_byte(int k) { return 3 - (k >> 1); }
__device__ __forceinline__ uint32_t right_word(int k, uint32_t e, uint32_t o) { return k & 1 ? o : e; }
__device__ __forceinline__ uint32_t left_word(int k, uint32_t e, uint32_t o) { return k & 1 ? e : o; }

// acc + the signed byte b of word.
__device__ __forceinline__ uint32_t add_byte(uint32_t word, int b, uint32_t acc) {
  return (uint32_t)__dp4a((int)word, 1 << (8 * b), (int)acc);
}

// SPARSE: the setup for targets whose buckets hold few positions, where a
// 128-hit tile spans many query positions (10-20 Mbp bins): a lane per
// position instead of per (position, seed) pair.  The engine picks it from
// the target's average bucket size.  GENERAL: see CostTable.
template <bool SPARSE, bool GENERAL>
__global__ void __launch_bounds__(kGateThreads, 4) gate2_kernel(const __grid_constant__ Gate2Args a2) {
  const GateArgs &a = a2.g;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (a.tot->status & 4u) return;  // no tile table: the host reruns the wave with a larger one
  const uint32_t tile = a2.tile;
  unsigned char *mine = smem_raw + (threadIdx.x >> 5) * (sizeof(GateWarp) + tile * sizeof(uint4));
  GateWarp &wt = *reinterpret_cast<GateWarp *>(mine);
  uint4 *const slot = reinterpret_cast<uint4 *>(mine + sizeof(GateWarp));
  const uint32_t lane = threadIdx.x & 31;
  const CostTable<GENERAL> tab(a.sub);
  const uint32_t thr = 0x7FFFu - (uint32_t)a.xdrop;  // drawdown + thr has bit 15 set when it exceeds xdrop
  const uint32_t thr2 = thr * 0x10001u;
  const bool soft = ((a2.ref[0].w | a2.qry[0].w) & a2.soft_codes) != 0;
  unsigned long long cells_acc = 0;
  const unsigned long long total = a.tot->hits;
  const uint32_t nz = a.tot->nz;
  const WaveIn &w = a.w;

  // the tile the cursor hands hits out of (warp-uniform)
  unsigned long long h0 = 0;
  uint32_t nt = 0, cursor = 0;
  bool tiles_done = false;
  // the next tile's index, claimed from the work queue once half of the
  // current tile is handed out so that its latency is hidden (lane 0 holds it)
  bool claimed = false;
  unsigned long long claim = 0;
  // The tile setup spreads a tile's (position, seed) pairs over the lanes:
  // 32 / per_pos positions per pass, lane l on seed l % per_pos of position
  // l / per_pos, so all bucket bounds of a pass are loaded at once.
  const uint32_t per = w.per_pos, ppi = 32u / per, lpi = lane / per, lvar = lane - lpi * per;
  bool hdr = false;  // the claimed tile's header is on its way into wt.hdr
  auto put_slot = [&](uint32_t sl, uint32_t bst, uint32_t qa, uint32_t c, const CallDev &cd) {
    slot[sl] = make_uint4(bst - sl, qa, c,
                          min(cd.qoff + cd.qlen - qa, 0xFFFFu) | min(qa - cd.qoff, 0xFFFFu) << 16);
    atomicOr(&wt.bits[sl >> 5], 1u << (sl & 31u));
  };
  // Takes the next tile from the work queue and finds its slots.  Every lane
  // takes part; lanes busy with an earlier tile's hits hold what they need of
  // them in registers.
  auto next_tile = [&]() {
    unsigned long long j = claim;
    if (!claimed && lane == 0) j = atomicAdd(&a.tot->tiles, 1ull);
    j = __shfl_sync(0xffffffffu, j, 0);
    const bool have_hdr = claimed && hdr;
    claimed = false;
    hdr = false;
    h0 = j * (unsigned long long)tile;
    cursor = 0;
    if (h0 >= total) {
      tiles_done = true;
      nt = 0;
      return;
    }
    nt = (uint32_t)min((unsigned long long)tile, total - h0);
    uint32_t k0, k1, c0;
    if (have_hdr) {
      cp_async_wait_all();
      __syncwarp();
      k0 = wt.hdr[0];
      k1 = wt.hdr[1];
      c0 = wt.hdr[2];
    } else {
      k0 = a.tile_first[j];
      k1 = a.tile_first[j + 1];
      c0 = a.tile_call[j];
    }
    // positions k0 .. kend cover the tile (k1, the next tile's first
    // position, only if its hits start inside this one; the overlap test
    // below sorts that out)
    const uint32_t kend = min(k1, nz - 1);
    const CallDev call0 = w.calls[c0];
    const uint32_t next_off = c0 + 1 < w.ncalls ? w.calls[c0 + 1].pos_off : 0xFFFFFFFFu;
    __syncwarp();  // every lane has read what it needs of the previous tile
    if (lane < kMaxTile / 32) wt.bits[lane] = 0;
    __syncwarp();
    if constexpr (SPARSE) {
      // a lane per position, its seeds' bucket bounds loaded five at a time
      // (more would spill in this register budget)
      for (uint32_t k = k0 + lane; k <= kend; k += 32) {
        const uint32_t p = a.np_pos[k];
        unsigned long long lo = a.np_excl[k];
        uint32_t kmer, qpos, c = c0;
        CallDev cd = call0;
        if (p >= next_off) {  // the tile reaches into a later call
          while (c + 1 < w.ncalls && w.calls[c + 1].pos_off <= p) c++;
          cd = w.calls[c];
        }
        if (a.np_kmer && !w.seeds) {
          kmer = a.np_kmer[k];
          qpos = cd.start + (p - cd.pos_off);
        } else {
          position_seed(w, cd, p, &qpos, &kmer);
        }
        const uint32_t qa = cd.qoff + qpos + w.shape.size;
        constexpr uint32_t kBatch = 5;
        for (uint32_t v0 = 0; v0 < per; v0 += kBatch) {
          uint32_t beg[kBatch], cnt[kBatch];
#pragma unroll
          for (uint32_t u = 0; u < kBatch; u++) {
            cnt[u] = 0;
            beg[u] = 0;
            if (v0 + u < per) cnt[u] = bucket(w, seed_variant(kmer, v0 + u), &beg[u]);
          }
#pragma unroll
          for (uint32_t u = 0; u < kBatch; u++) {
            const unsigned long long hi = lo + cnt[u];
            if (cnt[u] && hi > h0 && lo < h0 + nt) {
              const unsigned long long first = lo > h0 ? lo : h0;
              put_slot((uint32_t)(first - h0), beg[u] + (uint32_t)(first - lo), qa, c, cd);
            }
            lo = hi;
          }
        }
      }
    } else {
      for (uint32_t kb = k0; kb <= kend; kb += ppi) {
        const uint32_t k = kb + lpi;
        const bool act = lpi < ppi && k <= kend;
        uint32_t cnt = 0, beg = 0, qa = 0, c = c0;
        unsigned long long lo = 0;
        CallDev cd = call0;
        if (act) {
          const uint32_t p = a.np_pos[k];
          lo = a.np_excl[k];
          uint32_t kmer, qpos;
          if (p >= next_off) {  // the tile reaches into a later call
            while (c + 1 < w.ncalls && w.calls[c + 1].pos_off <= p) c++;
            cd = w.calls[c];
          }
          if (a.np_kmer && !w.seeds) {
            kmer = a.np_kmer[k];
            qpos = cd.start + (p - cd.pos_off);
          } else {
            position_seed(w, cd, p, &qpos, &kmer);
          }
          qa = cd.qoff + qpos + w.shape.size;
          cnt = bucket(w, seed_variant(kmer, lvar), &beg);
        }
        // the position's earlier seeds' hits come first: inclusive scan of the
        // counts over the position's lanes
        uint32_t incl = cnt;
#pragma unroll
        for (uint32_t d = 1; d < 32; d <<= 1) {
          const uint32_t up = __shfl_up_sync(0xffffffffu, incl, d);
          if (lvar >= d) incl += up;
        }
        if (cnt) {
          lo += incl - cnt;
          const unsigned long long hi = lo + cnt;
          if (hi > h0 && lo < h0 + nt) {
            const unsigned long long first = lo > h0 ? lo : h0;
            put_slot((uint32_t)(first - h0), beg + (uint32_t)(first - lo), qa, c, cd);
          }
        }
      }
    }
    __syncwarp();
    {  // the last slot start before each 32 hits
      const uint32_t b = lane < kMaxTile / 32 ? wt.bits[lane] : 0u;
      uint32_t top = b ? 32u * lane + 31u - (uint32_t)__clz((int)b) : 0u;
#pragma unroll
      for (uint32_t d = 1; d < kMaxTile / 32; d <<= 1) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, top, d);
        if (lane >= d) top = max(top, up);
      }
      top = __shfl_up_sync(0xffffffffu, top, 1);
      if (lane < kMaxTile / 32) wt.carry[lane] = lane ? top : 0u;
    }
    __syncwarp();
  };

  // The tile's next 32 hits, one per lane (the reference position and the
  // slot), loaded a round before lanes take them.
  uint32_t pos_next = 0, slot_next = 0;
  auto fetch_hits = [&]() {
    const uint32_t t = cursor + lane;
    if (t < nt) {
      const uint32_t b = wt.bits[t >> 5] & (0xFFFFFFFFu >> (31u - (t & 31u)));
      slot_next = b ? (t & ~31u) + 31u - (uint32_t)__clz((int)b) : wt.carry[t >> 5];
      pos_next = __ldg(w.pos_table + (slot[slot_next].x + t));
    }
  };

  // Lane state: its hit (anchors, call, index in the wave); the directions
  // scored this round (act) and the one that waits for its turn; how far from
  // the anchor the round's window stands; cells left to the edge or the cap
  // per direction (right low half, left high half) and whether that is the
  // cap; drawdowns at the round's start (halves); the summed bounds of the
  // maxima; cells scored.
  bool have = false, wait_left = false, cap_r = false, cap_l = false;
  uint32_t act = 0, hr0 = 0, hq0 = 0, hcall = 0, left = 0, draw = 0, cells = 0;
  int32_t off = 0, bound = 0;
  unsigned long long hidx = 0;
  constexpr uint32_t kGoRight = 1, kGoLeft = 2;

  while (true) {
    if (!claimed && !tiles_done && 2 * cursor >= nt) {
      if (lane == 0) claim = atomicAdd(&a.tot->tiles, 1ull);
      claimed = true;
    } else if (claimed && !hdr) {
      // a round after the claim: the claimed tile's header, copied into
      // shared memory while this round is scored
      const unsigned long long jn = __shfl_sync(0xffffffffu, claim, 0);
      if (jn * (unsigned long long)tile < total && lane < 3)
        cp_async4(&wt.hdr[lane], lane == 0 ? a.tile_first + jn : lane == 1 ? a.tile_first + jn + 1 : a.tile_call + jn);
      cp_async_commit();
      hdr = true;
    }
    // lanes without a hit take the tile's next ones; when the tile runs out
    // the next one is set up at once, so that no round runs half empty
    unsigned need = __ballot_sync(0xffffffffu, !have);
    while (need && !tiles_done) {
      if (cursor >= nt) {
        next_tile();
        if (tiles_done) break;
        fetch_hits();
      }
      const uint32_t rank = (uint32_t)__popc(need & lanemask_lt());
      const uint32_t sl = __shfl_sync(0xffffffffu, slot_next, rank);
      const uint32_t pos = __shfl_sync(0xffffffffu, pos_next, rank);
      if (!have && cursor + rank < nt) {
        const uint4 s = slot[sl];
        have = true;
        hr0 = pos + w.shape.size;
        hq0 = s.y;
        hcall = s.z;
        hidx = h0 + cursor + rank;
        const uint32_t er = min(w.rlen - hr0, s.w & 0xFFFFu), el = min(hr0, s.w >> 16);
        cap_r = er > a.cap;
        cap_l = el > a.cap;
        left = min(er, a.cap) | min(el, a.cap) << 16;
        act = kGoRight | kGoLeft;
        wait_left = false;
        off = 0;
        draw = 0;
        bound = 0;
        cells = 0;
      }
      cursor = min(cursor + (uint32_t)__popc(need), nt);
      __syncwarp();
      fetch_hits();
      need = __ballot_sync(0xffffffffu, !have);
    }
    if (!__any_sync(0xffffffffu, have)) break;  // no hits left in the queue
    // an idle lane scores the first window of each sequence
    const uint32_t vr = have ? hr0 + (uint32_t)off : (uint32_t)kLeft, vq = have ? hq0 + (uint32_t)off : (uint32_t)kLeft;
    if (!have) act = 0;
    uint32_t Rc[kWinChunks], Qc[kWinChunks], sp[3];
    {
      const uint4 *rp = a2.ref + ((vr + (64 - kLeft)) >> 5), *qp = a2.qry + ((vq + (64 - kLeft)) >> 5);
      uint4 rr[4], qr[4];
#pragma unroll
      for (int i = 0; i < 4; i++) rr[i] = __ldg(rp + i);
#pragma unroll
      for (int i = 0; i < 4; i++) qr[i] = __ldg(qp + i);
      uint32_t rs[3], qs[3];
      window_codes(rr, vr, Rc, rs);
      window_codes(qr, vq, Qc, qs);
#pragma unroll
      for (int i = 0; i < 3; i++) sp[i] = rs[i] | qs[i];
    }
    uint2 sel[kWinChunks];
#pragma unroll
    for (int c = 0; c < kWinChunks; c++) {
      sel[c] = CostTable<GENERAL>::index(Rc[c], Qc[c]);
      wt.sel[c][lane] = sel[c];
    }
    // Every lane scores the whole window.  Per eight-cell group it keeps the
    // drawdowns before the group and flags the group when its largest cost
    // minus the minimum exceeds xdrop (no flag: no cell of the group
    // dropped).  Flags: left group g at bit 31 - g, right group g at bit
    // 15 - kSolo - g.
    uint32_t flags = 0;
    uint32_t m2, P;
    {
      uint32_t Ar = kCostBase + (draw & 0xFFFFu), Al = kCostBase + (draw >> 16), ml = kCostBase;
#pragma unroll
      for (int g = 0; g < kSolo; g++) {  // the left extension's first groups
        const int f = kGroupsL - 1 - g;  // the group's place in the window
        const uint32_t e = tab.costs((f & 1) ? sel[f >> 1].x >> 16 : sel[f >> 1].x),
                       o = tab.costs((f & 1) ? sel[f >> 1].y >> 16 : sel[f >> 1].y);
        wt.grp[g][lane] = (Al - ml + thr) << 16;
        uint32_t hi = 0;
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
          const uint32_t A1 = add_byte(left_word(k, e, o), left_byte(k), Al);
          Al = add_byte(left_word(k + 1, e, o), left_byte(k + 1), A1);
          ml = (uint32_t)__vimin3_s32((int)ml, (int)A1, (int)Al);
          hi = (uint32_t)__vimax3_s32((int)hi, (int)A1, (int)Al);
        }
        flags |= ((hi - ml + thr) & 0x8000u) << (16 - g);
      }
      m2 = ml << 16 | kCostBase;
      P = Al * 0x10000u + Ar;
#pragma unroll
      for (int g = 0; g < kGroupsR; g++) {
        const int fl = kGroupsL - 1 - kSolo - g, fr = kGroupsL + g;
        const uint32_t le = tab.costs((fl & 1) ? sel[fl >> 1].x >> 16 : sel[fl >> 1].x),
                       lo = tab.costs((fl & 1) ? sel[fl >> 1].y >> 16 : sel[fl >> 1].y),
                       re = tab.costs((fr & 1) ? sel[fr >> 1].x >> 16 : sel[fr >> 1].x),
                       ro = tab.costs((fr & 1) ? sel[fr >> 1].y >> 16 : sel[fr >> 1].y);
        wt.grp[g + kSolo][lane] = P - m2 + thr2;
        uint32_t hi = 0;
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
          const uint32_t Al1 = add_byte(left_word(k, le, lo), left_byte(k), Al);
          const uint32_t Ar1 = add_byte(right_word(k, re, ro), right_byte(k), Ar);
          Al = add_byte(left_word(k + 1, le, lo), left_byte(k + 1), Al1);
          Ar = add_byte(right_word(k + 1, re, ro), right_byte(k + 1), Ar1);
          const uint32_t P1 = Al1 * 0x10000u + Ar1;
          P = Al * 0x10000u + Ar;
          m2 = __vimin3_u16x2(m2, P1, P);
          hi = __vimax3_u16x2(hi, P1, P);
        }
        flags |= ((hi - m2 + thr2) & 0x80008000u) >> (g + kSolo);
      }
    }
    // The first dropping cell of each direction (kRight, kLeft: none): the
    // eight cells of its first flagged group, both directions at once.  A
    // drawdown runs biased by thr, floored at it, and shows in bit 15.  When
    // seven largest scores can exceed xdrop a flag may be loose (the minimum
    // fell after the drawdown): the next flagged group is looked at then.
    __syncwarp();
    uint32_t drop_r = kRight, drop_l = kLeft;
    uint32_t todo = flags & ((act & kGoRight ? 0xFFFFu : 0u) | (act & kGoLeft ? 0xFFFF0000u : 0u));
    while (__any_sync(0xffffffffu, todo != 0)) {
      const uint32_t tl = todo & 0xFFFF0000u, tr = todo << 16;
      const uint32_t gl = tl ? (uint32_t)__clz((int)tl) : 0u, gr = tr ? (uint32_t)__clz((int)tr) - kSolo : 0u;
      const uint32_t fl = kGroupsL - 1 - gl, fr = kGroupsL + gr;
      const uint2 wl = wt.sel[fl >> 1][lane], wr = wt.sel[fr >> 1][lane];
      const uint32_t shl = (fl & 1u) << 4, shr = (fr & 1u) << 4;
      const uint32_t le = tab.costs(wl.x >> shl), lo = tab.costs(wl.y >> shl), re = tab.costs(wr.x >> shr),
                     ro = tab.costs(wr.y >> shr);
      uint32_t E = permute(wt.grp[gr + kSolo][lane], wt.grp[gl][lane], 0x7610u);
      uint32_t F = 0;  // bits 15 and 31: the direction has dropped
      int32_t after = 0;  // -128 * (cells from the drop on, right + 16 * left)
#pragma unroll
      for (int k = 0; k < 8; k++) {
        // both cells' costs, sign-extended to 16 bits
        const uint32_t rb = (uint32_t)right_byte(k), lb = 4u + (uint32_t)left_byte(k);
        const uint32_t c2 = permute(right_word(k, re, ro), left_word(k, le, lo),
                                        rb | (8u | rb) << 4 | lb << 8 | (8u | lb) << 12);
        E = __viaddmax_u16x2(E, c2, thr2);
        F = (F | E) & 0x80008000u;
        after = __dp4a((int)F, 0x10000100, after);
      }
      const uint32_t n = (uint32_t)(-after) >> 7, n_r = n & 15u, n_l = n >> 4;
      if (tr) {
        if (n_r) drop_r = 8 * gr + 8 - n_r;
        todo = n_r ? todo & 0xFFFF0000u : todo & ~(0x8000u >> (gr + kSolo));
      }
      if (tl) {
        if (n_l) drop_l = 8 * gl + 8 - n_l;
        todo = n_l ? todo & 0xFFFFu : todo & ~(0x80000000u >> gl);
      }
    }
    __syncwarp();
    // the first special base on each side (kRight, kLeft: none)
    uint32_t sp_r, sp_l;
    {
      static_assert(kLeft == 56, "the special words below split at base 56");
      const uint32_t r0 = __funnelshift_r(sp[1], sp[2], 24), r1 = sp[2] >> 24;
      const uint32_t l0 = __funnelshift_l(sp[0], sp[1], 8), l1 = sp[0] << 8;
      sp_r = r0 ? (uint32_t)__ffs((int)r0) - 1u : r1 ? 31u + (uint32_t)__ffs((int)r1) : (uint32_t)kRight;
      sp_l = l0 ? (uint32_t)__clz((int)l0) : l1 ? 32u + (uint32_t)__clz((int)l1) : (uint32_t)kLeft;
    }
    // How each direction ends: a drop, a special base, the edge or the cap --
    // or not in this round.
    const uint32_t left_r = left & 0xFFFFu, left_l = left >> 16;
    const uint32_t lim_r = min(left_r, (uint32_t)kRight), lim_l = min(left_l, (uint32_t)kLeft);
    const bool ar = (act & kGoRight) != 0, al = (act & kGoLeft) != 0;
    const bool dr = drop_r < min(lim_r, sp_r), dl = drop_l < min(lim_l, sp_l);
    const bool sr = !dr && sp_r < lim_r, sl = !dl && sp_l < lim_l;
    const bool er = !dr && !sr && left_r <= (uint32_t)kRight, el = !dl && !sl && left_l <= (uint32_t)kLeft;
    const bool more_r = ar && !dr && !sr && !er, more_l = al && !dl && !sl && !el;
    bool exact = (ar && er && cap_r) || (al && el && cap_l);  // past the cap
    if (soft && ((ar && sr) || (al && sl))) {  // a special base that may not end the extension
      int32_t worst = (int32_t)0x80000000;
      if (ar && sr) worst = a.sub[w.ref[vr + sp_r] * kNuc + w.qbuf[vq + sp_r]];
      if (al && sl) worst = max(worst, a.sub[w.ref[vr - 1u - sp_l] * kNuc + w.qbuf[vq - 1u - sp_l]]);
      exact |= (long long)worst + a.xdrop >= 0;
    }
    if (ar) {
      cells += dr ? drop_r + 1 : sr ? sp_r + 1 : lim_r;
      bound += (int32_t)(kCostBase - (m2 & 0xFFFFu));
    }
    if (al) {
      cells += dl ? drop_l + 1 : sl ? sp_l + 1 : lim_l;
      bound += (int32_t)(kCostBase - (m2 >> 16));
    }
    if (have) {
      if (!exact && (more_r || more_l || wait_left)) {  // another round for this hit
        const uint32_t m = (ar ? 0xFFFFu : 0u) | (al ? 0xFFFF0000u : 0u);
        draw = ((P - m2) & m) | (draw & ~m);
        if (more_l) left -= (uint32_t)kLeft << 16;
        if (more_r) {  // the right extension first; the left one waits if it goes on as well
          left -= kRight;
          wait_left |= more_l;
          act = kGoRight;
          off += kRight;
        } else {
          // to the left: from where its first round ended, or on from there
          off = wait_left ? -kLeft : off - kLeft;
          wait_left = false;
          act = kGoLeft;
        }
      } else {
        const bool maybe = a.total_exact ? bound >= a.hspthresh
                                         : sat_i32((double)__int2float_rn(bound)) >= a.hspthresh;
        if (exact || maybe) {
          const uint32_t at = atomicAdd(&a.tot->cand, 1u);
          if (at < a.cand_cap)
            a.cand[at] = Cand{scope_of(a.scope_lo, min(a.tot->n_scopes, a.scope_cap), hidx), hr0, hq0,
                              hcall | kLongFlag, 0, 0};
        } else {
          cells_acc += cells;
        }
        have = false;
      }
    }
  }
  for (int d = 16; d > 0; d >>= 1) cells_acc += __shfl_down_sync(0xffffffffu, cells_acc, d);
  if (lane == 0 && cells_acc) atomicAdd(&a.tot->cells, cells_acc);
}

}  // namespace hz
