// Lockstep score gate over 2-bit packed sequences (included by hz_wave.cuh).
//
// The same work as gate_kernel -- fused hit expansion and the X-drop score
// bound of every hit, src/gpu/kernels.rs:521-1057 -- organised so that a
// warp's 32 lanes run one instruction stream:
//   * a warp takes 32 hits of its tile at a time, a lane each, and scores both
//     extensions of each in one round over one window of each sequence, kLeft
//     bases before the anchor and kRight after it.  Random hits end after ~40
//     cells to the left (19 of them the seed) and ~21 to the right, so one
//     round ends 92 % of the hits; those that go on wait in a ring until 32
//     have gathered for another round from where they stand;
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
// Measured, ps per hit against a 200 Mbp target (5.4e9 hits) / a 10 Mbp bin: a
// kernel of one direction per round over two packed copies, a shared-memory
// lookup and three adds per cell took 60.1 / 68; this one, with the 8 % that
// go on keeping their lanes, 36.5 / 47; with the ring, which leaves the first
// round without per-lane state, 33.7 / 42; with a tile's bucket bounds loaded
// together and 256-hit tiles, 28.0 / 35.  ncu: issue 81 %, ALU 71 %, L1 72 %.
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
// Blocks of four warps, seven per SM: 72 registers a thread.  At 64 registers
// (32 warps) the compiler rebuilds constants and addresses, 806 instructions
// per round instead of 730, and 24 warps at 80 registers leave the issue slots
// empty: 27.97 ps per hit against 29.9 and 29.0 (200 Mbp target, 256-hit
// tiles).
constexpr int kGate2Threads = 128;
constexpr int kGate2Warps = kGate2Threads / 32;
constexpr int kGate2BlocksPerSm = 7;
// Running costs are kept as kCostBase + A in 16 unsigned bits (kWide: as
// Gate2Args::cost_base + A).  A falls by at most kLeft times the largest score
// in a round and rises by at most kLeft times the largest cost above the base
// + xdrop; a direction that has ended starts later rounds at the base.
constexpr uint32_t kCostBase = kLeft * 128;
static_assert(kWindow == 96, "a window is read as four 32-base records, at any offset in the first");
static_assert(kLeft % 8 == 0 && kRight % 8 == 0 && kLeft > kRight, "groups of eight cells; the left extension is longer");
// The largest xdrop the 16-bit halves hold: the drop test adds 0x7FFF - xdrop
// to a drawdown and reads bit 15, and the rescoring takes that word down by
// up to 128 per cell.
constexpr int32_t kGate2MaxXdrop = 32767 - 128;

// Hits of a wave of several calls, whatever its limit: the lockstep gate keeps
// a hit's index / 32 in 32 bits.  (A call alone has fewer than 2^32.)
constexpr uint64_t kMaxWaveHits = 1ull << 37;

// Shared memory of one warp; the slot arrays follow, 12 bytes per hit of a
// tile: 5.6 KB with 256-hit tiles, 164 KB per SM, which leaves 88 KB of L1.
// 128-hit tiles take 29.7 ps per hit (a setup every four rounds, mostly
// latency), 64-hit ones 34.1.
struct GateWarp {
  uint2 sel[kWinChunks][32];    // each lane's table indices: of the even and the odd cells of 16 bases
  uint32_t grp[kGroupsL][32];   // drawdowns before each group, biased (right low half, left high half)
  uint32_t bits[kMaxTile / 32];   // tile hits at which a slot starts
  uint32_t carry[kMaxTile / 32];  // the last slot that starts before the 32 hits
  uint32_t hdr[3];              // the claimed next tile's first position, the position after it, its call
  uint32_t nz;                  // positions with hits, and hits, of the wave
  unsigned long long total;
};
inline size_t gate2_smem(int tile) { return kGate2Warps * (sizeof(GateWarp) + (size_t)tile * 12); }

// Hits that go on for another round (8 % of them) wait in a ring of their
// warp in device memory, a word per field, fields kRingCap apart.  A round
// adds at most 32, and 32 are taken as soon as the ring holds them, so at most
// 31 + 32 wait.
constexpr uint32_t kRingCap = 64;
enum RingField : uint32_t {
  kRingR, kRingQ,  // anchors
  kRingCall,
  kRingHit,        // wave index / 32; the rest of it is in kRingState
  kRingOff,        // how far from the anchor the next window stands
  kRingDraw,       // drawdowns (right low half, left high half)
  kRingBound,      // summed bounds of the maxima so far
  kRingState,      // kGo*, kWaitLeft | wave index % 32 << 3 | cells scored so far << 8
  kRingFields
};
constexpr uint32_t kGoRight = 1, kGoLeft = 2;  // directions the next window scores
constexpr uint32_t kWaitLeft = 4;              // the left extension goes on after the right one
inline size_t gate2_ring_words(size_t blocks) { return blocks * kGate2Warps * kRingFields * kRingCap; }

struct Gate2Args {
  GateArgs g;
  // packed forward halves (pack2_kernel's records) from two records before
  // their first base: a window may start kLeft bases before the sequence.
  // Component w of the first record holds the non-ACGT codes of the sequence.
  const uint4 *ref, *qry;
  uint32_t *ring;       // gate2_ring_words words
  uint32_t tile;        // hits per warp tile, a multiple of 32, at most kMaxTile
  uint32_t soft_codes;  // bit c: code c (4..7) does not end every extension that meets it
  uint32_t cost_base;   // kLeft * (largest score), for kWide matrices
  int32_t min_total;    // the smallest total with (i32)(f32)total >= hspthresh
  const uint16_t *nbr_live;  // which seeds of a k-mer have hits (nbr_hits_kernel), or null
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

__device__ __forceinline__ uint32_t min_halves(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("min.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
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

// How a matrix's ACGT scores are looked up.  kAlike: complementary pairs score
// alike and costs fit a signed byte; kGeneral: any scores of a signed byte, whose
// tables hold the scores themselves, since the cost of -128 is no signed byte
// (sums negate them in the dot product's other factor, and the rescoring runs
// on complements, so that costs nothing); kWide: alike, costs of 16 bits.
enum CostMode : int { kAlike, kGeneral, kWide };

// The costs of eight cells: bytes of the even cells, of the odd cells (kAlike;
// kGeneral: of their scores); 16-bit pairs of cells 0 2, 4 6, 1 3, 5 7 (kWide).
template <int MODE> struct Cells8 {
  uint32_t w[MODE == kWide ? 4 : 2];
};

// Costs (negated scores) of ACGT pairs.  The index of a pair is reference ^
// query | parity << 2, parity the xor of the reference code's two bits: with
// A C G T = 0..3 a complement flips both bits, so a matrix with equal scores
// for complementary pairs -- HOXD70, and any matrix that treats the strands
// alike -- has one score per index, and eight bytes hold them.  kGeneral
// matrices add the reference code's low bit as bit 3 and hold a second table
// for it; kWide ones look low and high bytes up apart and pair them, three
// more permutes for four cells (a close-species score set, mismatches down to
// -356, 68 M hits against a 10 Mbp bin: 3.7 ms in the lane-refill gate, 2.5
// here).
template <int MODE>
struct CostTable {
  uint32_t t[MODE == kAlike ? 2 : 4];
  __device__ __forceinline__ explicit CostTable(const int32_t *sub) {
#pragma unroll
    for (int i = 0; i < (MODE == kAlike ? 2 : 4); i++) {
      t[i] = 0;
#pragma unroll
      for (int x = 0; x < 4; x++) {
        const int low = MODE == kGeneral ? i >> 1 : 0, parity = i & 1;
        const int r = (parity ^ low) << 1 | low;
        const int32_t score = sub[r * kNuc + (r ^ x)];
        const uint32_t cost = (uint32_t)(MODE == kGeneral ? score : -score);
        t[i] |= (cost >> (MODE == kWide && i >= 2 ? 8 : 0) & 0xFFu) << (8 * x);
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
    if (MODE == kGeneral) {
      e.x |= (r & 0x11111111u) << 3;
      e.y |= (r << 1) & 0x88888888u;
    }
    return e;
  }
  // The cost bytes of the four cells whose indices are the low nibbles of s.
  __device__ __forceinline__ uint32_t bytes(uint32_t s) const {
    if (MODE != kGeneral) return permute(t[0], t[1], s);
    const uint32_t lo = s & 0x7777u;
    // bit 3 of each nibble as a byte mask: nibble 9 takes the sign of byte 1
    const uint32_t m = permute(0x00008000u, 0u, ((s >> 3) & 0x1111u) * 9u);
    return (permute(t[0], t[1], lo) & ~m) | (permute(t[MODE == kAlike ? 0 : 2], t[MODE == kAlike ? 1 : 3], lo) & m);
  }
  // The costs of eight cells from the indices of the even and the odd ones.
  __device__ __forceinline__ Cells8<MODE> cells(uint32_t even, uint32_t odd) const {
    Cells8<MODE> c;
    if constexpr (MODE == kWide) {
      const uint32_t el = permute(t[0], t[1], even), eh = permute(t[2], t[3], even);
      const uint32_t ol = permute(t[0], t[1], odd), oh = permute(t[2], t[3], odd);
      c.w[0] = permute(el, eh, 0x5140u);
      c.w[1] = permute(el, eh, 0x7362u);
      c.w[2] = permute(ol, oh, 0x5140u);
      c.w[3] = permute(ol, oh, 0x7362u);
    } else {
      c.w[0] = bytes(even);
      c.w[1] = bytes(odd);
    }
    return c;
  }
};

// Of base b (0..7) of a group: the word of its cost, and the byte or half.
template <int MODE> __device__ __forceinline__ uint32_t cost_word(const Cells8<MODE> &c, int b) {
  return MODE == kWide ? c.w[MODE == kWide ? (b & 1) * 2 + (b >> 2) : 0] : c.w[b & 1];
}
// acc + the cost of base b.
template <int MODE> __device__ __forceinline__ uint32_t add_cost(const Cells8<MODE> &c, int b, uint32_t acc) {
  if (MODE == kWide) return (uint32_t)__dp2a_lo((int)cost_word(c, b), b & 2 ? 0x100 : 1, (int)acc);
  return (uint32_t)__dp4a((int)cost_word(c, b), (int)((MODE == kGeneral ? 0xFFu : 1u) << (8 * (b >> 1))), (int)acc);
}
// The costs (kGeneral: the scores) of base br of one group and base bl of
// another, as 16-bit halves.
template <int MODE>
__device__ __forceinline__ uint32_t cost_pair(const Cells8<MODE> &r, int br, const Cells8<MODE> &l, int bl) {
  uint32_t s;
  if (MODE == kWide) {
    const uint32_t x = br & 2u, y = 4u + (bl & 2u);
    s = x | (x + 1) << 4 | y << 8 | (y + 1) << 12;
  } else {
    const uint32_t x = (uint32_t)br >> 1, y = 4u + ((uint32_t)bl >> 1);
    s = x | (8u | x) << 4 | y << 8 | (8u | y) << 12;
  }
  return permute(cost_word(r, br), cost_word(l, bl), s);
}

// SPARSE: the setup for targets whose buckets hold few positions, where a
// tile spans many query positions (10-20 Mbp bins): a lane per
// position instead of per (position, seed) pair.  The engine picks it from
// the target's average bucket size.  MODE: see CostMode.
template <bool SPARSE, int MODE>
__global__ void __launch_bounds__(kGate2Threads, kGate2BlocksPerSm) gate2_kernel(const __grid_constant__ Gate2Args a2) {
  const GateArgs &a = a2.g;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (a.tot->status & 4u) return;  // no tile table, or too many hits: the host reruns the wave, or its parts
  const uint32_t tile = a2.tile;
  unsigned char *mine = smem_raw + (threadIdx.x >> 5) * (sizeof(GateWarp) + tile * 12);
  GateWarp &wt = *reinterpret_cast<GateWarp *>(mine);
  // A slot is a run of tile hits of one (position, seed), stored at its first
  // hit: its pos_table index less that hit (so hit t is slot_x + t), the query
  // anchor (absolute) and the call.
  uint32_t *const slot_x = reinterpret_cast<uint32_t *>(mine + sizeof(GateWarp));
  uint32_t *const slot_q = slot_x + tile, *const slot_call = slot_q + tile;
  const uint32_t lane = threadIdx.x & 31;
  const CostTable<MODE> tab(a.sub);
  const uint32_t cost_base = MODE == kWide ? a2.cost_base : kCostBase;
  const uint32_t thr = 0x7FFFu - (uint32_t)a.xdrop;  // drawdown + thr has bit 15 set when it exceeds xdrop
  const uint32_t thr2 = thr * 0x10001u;
  const bool soft = ((a2.ref[0].w | a2.qry[0].w) & a2.soft_codes) != 0;
  const WaveIn &w = a.w;
  uint32_t cells_acc = 0;  // cells of the lane's hits, added to the wave's count before it can wrap

  // the tile the cursor hands hits out of (warp-uniform); a wave has at most
  // kMaxWaveHits hits, so hit indices / 32 fit 32 bits
  uint32_t tile_at = 0, nt = 0, cursor = 0;
  // the next tile's index, claimed from the work queue once half of the
  // current tile is handed out so that its latency is hidden (lane 0 holds it)
  bool claimed = false;
  uint32_t claim = 0;
  // The tile setup spreads a tile's (position, seed) pairs over the lanes:
  // 32 / per_pos positions per pass, lane l on seed l % per_pos of position
  // l / per_pos, so all bucket bounds of a pass are loaded at once.
  const uint32_t per = w.per_pos, ppi = 32u / per, lpi = lane / per, lvar = lane - lpi * per;
  bool hdr = false;  // the claimed tile's header is on its way into wt.hdr
  auto put_slot = [&](uint32_t sl, uint32_t bst, uint32_t qa, uint32_t c) {
    slot_x[sl] = bst - sl;
    slot_q[sl] = qa;
    slot_call[sl] = c;
    atomicOr(&wt.bits[sl >> 5], 1u << (sl & 31u));
  };
  // Takes the next tile from the work queue and finds its slots, from as few
  // waits as it can (the positions, then their seeds' buckets); leaves nt 0
  // when there is none.
  auto next_tile = [&]() {
    if (!claimed && lane == 0) claim = (uint32_t)atomicAdd(&a.tot->tiles, 1ull);
    const uint32_t j = __shfl_sync(0xffffffffu, claim, 0);
    const bool have_hdr = claimed && hdr;
    claimed = false;
    hdr = false;
    const unsigned long long h0 = j * (unsigned long long)tile, total = wt.total;
    tile_at = j;
    cursor = 0;
    nt = 0;
    if (h0 >= total) return;
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
    const uint32_t kend = min(k1, wt.nz - 1);
    const CallDev call0 = w.calls[c0];
    const uint32_t next_off = c0 + 1 < w.ncalls ? w.calls[c0 + 1].pos_off : 0xFFFFFFFFu;
    __syncwarp();  // every lane has read what it needs of the previous tile
    if (lane < kMaxTile / 32) wt.bits[lane] = 0;
    __syncwarp();
    for (uint32_t kb = k0; kb <= kend; kb += 32) {
      // a lane per position: its first hit, k-mer, query anchor and call, with
      // one wait for all of them
      const uint32_t nk = min(kend - kb + 1, 32u);
      uint32_t kmer = 0, qa = 0, c = c0;
      unsigned long long lo = 0;
      if (lane < nk) {
        const uint32_t p = a.np_pos[kb + lane];
        lo = a.np_excl[kb + lane];
        CallDev cd = call0;
        if (p >= next_off) {  // the tile reaches into a later call
          while (c + 1 < w.ncalls && w.calls[c + 1].pos_off <= p) c++;
          cd = w.calls[c];
        }
        uint32_t qpos;
        if (a.np_kmer && !w.seeds) {
          kmer = a.np_kmer[kb + lane];
          qpos = cd.start + (p - cd.pos_off);
        } else {
          position_seed(w, cd, p, &qpos, &kmer);
        }
        qa = cd.qoff + qpos + w.shape.size;
      }
      if constexpr (SPARSE) {
        // A lane looks up its own position's seeds with hits, kBatch at a
        // time.  Most seeds of a sparse target have none (93 % at 1 Mbp, 55 %
        // at 10 Mbp), and a look at a bucket costs two loads a lane: 5.7 ps
        // from L2, 19 ps of random DRAM access from a 14-care pattern's 1 GB
        // table.  One 16-bit mask per position says which to look at: 1 Mbp
        // target 182 -> 120 us, 10 Mbp 34.8 -> 32.4 ps per hit, 14of22 and 50
        // Mbp 1046 -> 530 us.  3 to 7 at a time are within 3 %.
        constexpr uint32_t kBatch = 4;
        if (lane < nk) {
          uint32_t live = per > 1 && a2.nbr_live ? (uint32_t)__ldg(a2.nbr_live + kmer) : (1u << per) - 1u;
          while (live) {
            uint32_t beg[kBatch], cnt[kBatch];
#pragma unroll
            for (uint32_t u = 0; u < kBatch; u++) {
              cnt[u] = 0;
              beg[u] = 0;
              if (live) cnt[u] = bucket(w, seed_variant(kmer, (uint32_t)__ffs((int)live) - 1u), &beg[u]);
              live &= live - 1u;
            }
#pragma unroll
            for (uint32_t u = 0; u < kBatch; u++) {
              const unsigned long long hi = lo + cnt[u];
              if (cnt[u] && hi > h0 && lo < h0 + nt) {
                const unsigned long long first = lo > h0 ? lo : h0;
                put_slot((uint32_t)(first - h0), beg[u] + (uint32_t)(first - lo), qa, c);
              }
              lo = hi;
            }
          }
        }
      } else {
        // the lanes spread over (position, seed) pairs, the bucket bounds of
        // up to kPasses passes loaded before any is used
        constexpr uint32_t kPasses = 3;
        for (uint32_t b = 0; b < nk; b += kPasses * ppi) {
          uint32_t beg[kPasses], cnt[kPasses];
#pragma unroll
          for (uint32_t u = 0; u < kPasses; u++) {
            cnt[u] = 0;
            beg[u] = 0;
            if (b + u * ppi < nk) {
              const uint32_t src = b + u * ppi + lpi;
              const uint32_t km = __shfl_sync(0xffffffffu, kmer, src & 31u);
              if (lpi < ppi && src < nk) cnt[u] = bucket(w, seed_variant(km, lvar), &beg[u]);
            }
          }
#pragma unroll
          for (uint32_t u = 0; u < kPasses; u++) {
            if (b + u * ppi >= nk) break;
            const uint32_t src = (b + u * ppi + lpi) & 31u;
            // the position's earlier seeds' hits come first: inclusive scan of
            // the counts over the position's lanes
            uint32_t incl = cnt[u];
#pragma unroll
            for (uint32_t d = 1; d < 32; d <<= 1) {
              const uint32_t up = __shfl_up_sync(0xffffffffu, incl, d);
              if (lvar >= d) incl += up;
            }
            const unsigned long long at = __shfl_sync(0xffffffffu, lo, src) + (incl - cnt[u]);
            const uint32_t sq = __shfl_sync(0xffffffffu, qa, src), sc = __shfl_sync(0xffffffffu, c, src);
            if (cnt[u] && at + cnt[u] > h0 && at < h0 + nt) {
              const unsigned long long first = at > h0 ? at : h0;
              put_slot((uint32_t)(first - h0), beg[u] + (uint32_t)(first - at), sq, sc);
            }
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
  // slot), loaded while the hits before them are scored.
  uint32_t pos_next = 0, slot_next = 0;
  auto fetch_hits = [&]() {
    const uint32_t t = cursor + lane;
    if (t < nt) {
      const uint32_t b = wt.bits[t >> 5] & (0xFFFFFFFFu >> (31u - (t & 31u)));
      slot_next = b ? (t & ~31u) + 31u - (uint32_t)__clz((int)b) : wt.carry[t >> 5];
      pos_next = __ldg(w.pos_table + (slot_x[slot_next] + t));
    }
    if (!claimed && 2 * cursor >= nt) {
      if (lane == 0) claim = (uint32_t)atomicAdd(&a.tot->tiles, 1ull);
      claimed = true;
    } else if (claimed && !hdr) {
      // 32 hits after the claim: the claimed tile's header, copied into
      // shared memory while hits are scored
      const uint32_t jn = __shfl_sync(0xffffffffu, claim, 0);
      if (jn * (unsigned long long)tile < wt.total && lane < 3)
        cp_async4(&wt.hdr[lane], lane == 0 ? a.tile_first + jn : lane == 1 ? a.tile_first + jn + 1 : a.tile_call + jn);
      cp_async_commit();
      hdr = true;
    }
  };

  // Scores one window per lane from the drawdowns `draw`: the minima and last
  // costs of both extensions, one past the first drop of each direction (one
  // past the window: none), one past the first special base.  `between` runs
  // while the group states wait in shared memory.
  auto score = [&](uint32_t vr, uint32_t vq, uint32_t draw, uint32_t &m2, uint32_t &P, uint32_t &drop,
                   uint32_t &special, auto between) {
    uint32_t Rc[kWinChunks], Qc[kWinChunks];
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
      for (int i = 0; i < 3; i++) rs[i] |= qs[i];
      static_assert(kLeft == 56, "the special words below split at base 56");
      // the first set bit, among the next 32 when there is none (a bit past
      // the window stands for none at all)
      const uint32_t r0 = __funnelshift_r(rs[1], rs[2], 24), r1 = rs[2] >> 24 | 1u << (kRight - 32);
      const uint32_t l0 = __funnelshift_l(rs[0], rs[1], 8), l1 = rs[0] << 8 | 1u << (63 - kLeft);
      const uint32_t sp_r = (uint32_t)__clz((int)__brev(r0 ? r0 : r1)) + (r0 ? 1u : 33u);
      const uint32_t sp_l = (uint32_t)__clz((int)(l0 ? l0 : l1)) + (l0 ? 1u : 33u);
      special = sp_l << 16 | sp_r;
    }
    uint2 sel[kWinChunks];
#pragma unroll
    for (int c = 0; c < kWinChunks; c++) {
      sel[c] = CostTable<MODE>::index(Rc[c], Qc[c]);
      wt.sel[c][lane] = sel[c];
    }
    // Every lane scores the whole window.  Per eight-cell group it keeps the
    // drawdowns before the group and flags the group when its largest cost
    // minus the minimum exceeds xdrop (no flag: no cell of the group
    // dropped).  Flags: left group g at bit 31 - g, right group g at bit
    // 15 - kSolo - g.
    uint32_t flags = 0;
    {
      uint32_t Ar = cost_base + (draw & 0xFFFFu), Al = cost_base + (draw >> 16), ml = cost_base;
#pragma unroll
      for (int g = 0; g < kSolo; g++) {  // the left extension's first groups
        const int f = kGroupsL - 1 - g;  // the group's place in the window
        const Cells8<MODE> lc = tab.cells((f & 1) ? sel[f >> 1].x >> 16 : sel[f >> 1].x,
                                          (f & 1) ? sel[f >> 1].y >> 16 : sel[f >> 1].y);
        wt.grp[g][lane] = (Al - ml + thr) << 16;
        uint32_t hi = 0;
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
          const uint32_t A1 = add_cost(lc, 7 - k, Al);
          Al = add_cost(lc, 6 - k, A1);
          ml = (uint32_t)__vimin3_s32((int)ml, (int)A1, (int)Al);
          hi = (uint32_t)__vimax3_s32((int)hi, (int)A1, (int)Al);
        }
        flags |= ((hi - ml + thr) & 0x8000u) << (16 - g);
      }
      m2 = ml << 16 | cost_base;
      P = Al * 0x10000u + Ar;
#pragma unroll
      for (int g = 0; g < kGroupsR; g++) {
        const int fl = kGroupsL - 1 - kSolo - g, fr = kGroupsL + g;
        const Cells8<MODE> lc = tab.cells((fl & 1) ? sel[fl >> 1].x >> 16 : sel[fl >> 1].x,
                                          (fl & 1) ? sel[fl >> 1].y >> 16 : sel[fl >> 1].y);
        const Cells8<MODE> rc = tab.cells((fr & 1) ? sel[fr >> 1].x >> 16 : sel[fr >> 1].x,
                                          (fr & 1) ? sel[fr >> 1].y >> 16 : sel[fr >> 1].y);
        wt.grp[g + kSolo][lane] = P - m2 + thr2;
        uint32_t hi = 0;
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
          const uint32_t Al1 = add_cost(lc, 7 - k, Al);
          const uint32_t Ar1 = add_cost(rc, k, Ar);
          Al = add_cost(lc, 6 - k, Al1);
          Ar = add_cost(rc, k + 1, Ar1);
          const uint32_t P1 = Al1 * 0x10000u + Ar1;
          P = Al * 0x10000u + Ar;
          m2 = __vimin3_u16x2(m2, P1, P);
          hi = __vimax3_u16x2(hi, P1, P);
        }
        flags |= ((hi - m2 + thr2) & 0x80008000u) >> (g + kSolo);
      }
    }
    between();
    __syncwarp();
    // One past the first dropping cell of each direction: the eight cells of
    // its first flagged group, or of its last group when none is flagged, both
    // directions at once.  A drawdown runs biased by thr, floored at it, and
    // shows in bit 15; the cells from the drop on are counted, so none leaves
    // one past the window.  When seven largest scores can exceed xdrop a flag
    // may be loose (the minimum fell after the drawdown) and the next flagged
    // group is looked at.
    flags |= 0x80000000u >> (kGroupsL - 1) | 0x8000u >> (kGroupsL - 1);
    while (true) {
      // left group gl, right group gr - kSolo; their bases in the window
      const uint32_t gl = (uint32_t)__clz((int)flags), gr = (uint32_t)__clz((int)(flags << 16));
      const uint32_t fl = kGroupsL - 1 - gl, fr = kGroupsL - kSolo + gr;
      const uint2 wl = wt.sel[fl >> 1][lane], wr = wt.sel[fr >> 1][lane];
      const uint32_t shl = (fl & 1u) << 4, shr = (fr & 1u) << 4;
      const Cells8<MODE> lc = tab.cells(wl.x >> shl, wl.y >> shl), rc = tab.cells(wr.x >> shr, wr.y >> shr);
      uint32_t E = permute(wt.grp[gr][lane], wt.grp[gl][lane], 0x7610u);
      if (MODE == kGeneral) E = ~E;  // the complement falls by a cost as it rises by the score
      uint32_t F = 0;      // bits 15 and 31: the direction has dropped
      uint32_t after = 0;  // 128 * (cells from the drop on: right + 16 * left)
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const uint32_t pair = cost_pair(rc, k, lc, 7 - k);
        E = MODE == kGeneral ? __viaddmin_u16x2(E, pair, ~thr2) : __viaddmax_u16x2(E, pair, thr2);
        F = (F | (MODE == kGeneral ? ~E : E)) & 0x80008000u;
        after = __dp4a(F, 0x10000100u, after);
      }
      const uint32_t n = ((after >> 7) * 0x1001u) & 0x000F000Fu;  // the two counts in halves
      drop = gl * 0x80000u + gr * 8u + (9u << 16 | 9u) - 8u * kSolo - n;
      if (a.late_max_safe) break;
      const uint32_t loose = (gl < kGroupsL - 1 && !(n >> 16) ? 0x80000000u >> gl : 0u) |
                             (gr < kGroupsL - 1 && !(n & 0xFFFFu) ? 0x8000u >> gr : 0u);
      flags &= ~loose;
      if (!__any_sync(0xffffffffu, loose)) break;
    }
    __syncwarp();
  };

  // the warp's ring of waiting hits
  uint32_t *const ring = a2.ring + (size_t)(blockIdx.x * kGate2Warps + (threadIdx.x >> 5)) * (kRingFields * kRingCap);
  uint32_t ring_head = 0, ring_n = 0;
  // Adds the lanes' hits with `on` set to the ring.
  auto push = [&](bool on, uint32_t r0, uint32_t q0, uint32_t call, uint32_t hit, uint32_t off, uint32_t draw,
                  int32_t bound, uint32_t state) {
    const unsigned going = __ballot_sync(0xffffffffu, on);
    if (on) {
      uint32_t *to = ring + ((ring_head + ring_n + (uint32_t)__popc(going & lanemask_lt())) & (kRingCap - 1));
      to[kRingR * kRingCap] = r0;
      to[kRingQ * kRingCap] = q0;
      to[kRingCall * kRingCap] = call;
      to[kRingHit * kRingCap] = hit;
      to[kRingOff * kRingCap] = off;
      to[kRingDraw * kRingCap] = draw;
      to[kRingBound * kRingCap] = (uint32_t)bound;
      to[kRingState * kRingCap] = state;
    }
    ring_n += (uint32_t)__popc(going);
    __syncwarp();
  };
  // A hit that becomes a candidate.
  auto emit = [&](unsigned long long hit, uint32_t r0, uint32_t q0, uint32_t call) {
    const uint32_t at = atomicAdd(&a.tot->cand, 1u);
    if (at < a.cand_cap)
      a.cand[at] = Cand{scope_of(a.scope_lo, min(a.tot->n_scopes, a.scope_cap), hit), r0, q0, call | kLongFlag, 0, 0};
  };
  // Whether a special base that ends a direction (one past it: sp) may not do
  // so by its score alone.
  auto soft_end = [&](uint32_t r, uint32_t q) {
    return (long long)a.sub[w.ref[r] * kNuc + w.qbuf[q]] + a.xdrop >= 0;
  };
  constexpr uint32_t kMoreBias = (0x7FFFu - kLeft) << 16 | (0x7FFFu - kRight);  // sets a half's top bit past the window

  if (lane == 0) {
    wt.total = a.tot->hits;
    wt.nz = a.tot->nz;
  }
  __syncwarp();
  next_tile();
  if (nt) fetch_hits();
  while (true) {
    if (cells_acc >= 1u << 30) {
      atomicAdd(&a.tot->cells, (unsigned long long)cells_acc);
      cells_acc = 0;
    }
    if (ring_n < 32 && cursor < nt) {
      // 32 fresh hits of the tile; a lane without one scores the first window
      // of each sequence
      const bool have = cursor + lane < nt;
      const uint32_t hit = tile_at * (tile >> 5) + (cursor >> 5);
      const uint32_t vr = have ? pos_next + w.shape.size : (uint32_t)kLeft;
      const uint32_t vq = have ? slot_q[slot_next] : (uint32_t)kLeft, call = have ? slot_call[slot_next] : 0u;
      uint32_t m2, P, drop, special;
      score(vr, vq, 0u, m2, P, drop, special, [&]() {
        cursor += 32;
        if (cursor >= nt) next_tile();
        if (nt) fetch_hits();
      });
      // Cells scored: through the drop or the special base, to the edge or
      // the cap -- or more than the window holds, and the direction goes on.
      const CallDev cd = w.calls[call];
      const uint32_t er = min(w.rlen - vr, cd.qoff + cd.qlen - vq), el = min(vr, vq - cd.qoff);
      const uint32_t ends = min_halves(drop, special);
      const uint32_t use = min_halves(ends, min(er, a.cap) | min(el, a.cap) << 16);
      const uint32_t more = (use + kMoreBias) & 0x80008000u;
      const bool more_r = (more & 0x8000u) != 0, more_l = (int32_t)more < 0;
      bool exact = false;
      if (a.cap <= (uint32_t)kLeft)  // past the cap
        exact = (er > a.cap && a.cap <= (uint32_t)kRight && (use & 0xFFFFu) < (ends & 0xFFFFu)) ||
                (el > a.cap && (use >> 16) < (ends >> 16));
      if (soft && have) {
        const uint32_t sp_r = special & 0xFFFFu, sp_l = special >> 16;
        if (sp_r <= (uint32_t)kRight && sp_r == (use & 0xFFFFu)) exact |= soft_end(vr + sp_r - 1u, vq + sp_r - 1u);
        if (sp_l <= (uint32_t)kLeft && sp_l == use >> 16) exact |= soft_end(vr - sp_l, vq - sp_l);
      }
      const uint32_t cells = (use & 0xFFFFu) + (use >> 16) - (more_r ? 1u : 0u) - (more_l ? 1u : 0u);
      const int32_t bound = (int32_t)(2u * cost_base - (m2 & 0xFFFFu) - (m2 >> 16));
      const bool on = have && more && !exact;
      const bool cand = have && !on && (exact || bound >= a2.min_total);
      cells_acc += have && !on && !cand ? cells : 0u;
      if (cand) emit(hit * 32ull + lane, vr, vq, call);
      // the right extension goes on first; the left one waits if it does too
      push(on, vr, vq, call, hit, more_r ? (uint32_t)kRight : (uint32_t)-kLeft,
           (P - m2) & ((more_r ? 0xFFFFu : 0u) | (more_l ? 0xFFFF0000u : 0u)), bound,
           (more_r ? kGoRight | (more_l ? kWaitLeft : 0u) : kGoLeft) | lane << 3 | cells << 8);
    } else if (ring_n) {
      // up to 32 waiting hits, from where they stand
      const uint32_t n = min(ring_n, 32u);
      const bool have = lane < n;
      uint32_t r0 = kLeft, q0 = kLeft, call = 0, hit = 0, off = 0, was = 0, state = 0;
      int32_t bound = 0;
      if (have) {
        const uint32_t *at = ring + ((ring_head + lane) & (kRingCap - 1));
        r0 = at[kRingR * kRingCap];
        q0 = at[kRingQ * kRingCap];
        call = at[kRingCall * kRingCap];
        hit = at[kRingHit * kRingCap];
        off = at[kRingOff * kRingCap];
        was = at[kRingDraw * kRingCap];
        bound = (int32_t)at[kRingBound * kRingCap];
        state = at[kRingState * kRingCap];
      }
      ring_head += n;
      ring_n -= n;
      __syncwarp();  // every lane has its entry before new ones overwrite it
      const uint32_t vr = r0 + off, vq = q0 + off;
      const bool on_r = (state & kGoRight) != 0, on_l = (state & kGoLeft) != 0;
      uint32_t m2, P, drop, special;
      score(vr, vq, was, m2, P, drop, special, []() {});
      // cells left to the edge or the cap; a left extension that waits has
      // one window behind it
      const CallDev cd = w.calls[call];
      const uint32_t er = min(w.rlen - r0, cd.qoff + cd.qlen - q0), el = min(r0, q0 - cd.qoff);
      const uint32_t left_r = min(er, a.cap) - off, left_l = min(el, a.cap) + off;
      const uint32_t ends_r = min(drop & 0xFFFFu, special & 0xFFFFu), ends_l = min(drop >> 16, special >> 16);
      const uint32_t use_r = on_r ? min(ends_r, left_r) : 0u, use_l = on_l ? min(ends_l, left_l) : 0u;
      const bool more_r = use_r > (uint32_t)kRight, more_l = use_l > (uint32_t)kLeft;
      bool exact = (on_r && er > a.cap && use_r < ends_r && !more_r) || (on_l && el > a.cap && use_l < ends_l && !more_l);
      if (soft && have) {
        if (on_r && ends_r == (special & 0xFFFFu) && use_r == ends_r && !more_r)
          exact |= soft_end(vr + use_r - 1u, vq + use_r - 1u);
        if (on_l && ends_l == special >> 16 && use_l == ends_l && !more_l) exact |= soft_end(vr - use_l, vq - use_l);
      }
      const uint32_t cells = (state >> 8) + use_r + use_l - (more_r ? 1u : 0u) - (more_l ? 1u : 0u);
      bound += (int32_t)((on_r ? cost_base - (m2 & 0xFFFFu) : 0u) + (on_l ? cost_base - (m2 >> 16) : 0u));
      const bool waits = (state & kWaitLeft) != 0;
      const bool on = have && !exact && (more_r || more_l || waits);
      const bool cand = have && !on && (exact || bound >= a2.min_total);
      cells_acc += have && !on && !cand ? cells : 0u;
      if (cand) emit(hit * 32ull + (state >> 3 & 31u), r0, q0, call);
      const uint32_t m = (on_r ? 0xFFFFu : 0u) | (on_l ? 0xFFFF0000u : 0u);
      push(on, r0, q0, call, hit, more_r ? off + kRight : waits ? (uint32_t)-kLeft : off - kLeft,
           ((P - m2) & ((more_r ? 0xFFFFu : 0u) | (more_l ? 0xFFFF0000u : 0u))) | (was & ~m), bound,
           (more_r ? kGoRight | (state & kWaitLeft) : kGoLeft) | (state & 31u << 3) | cells << 8);
    } else {
      break;
    }
  }
  unsigned long long sum = cells_acc;
  for (int d = 16; d > 0; d >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, d);
  if (lane == 0 && sum) atomicAdd(&a.tot->cells, sum);
}

}  // namespace hz
