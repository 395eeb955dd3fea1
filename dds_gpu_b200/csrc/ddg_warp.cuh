// The search of one job by one warp: every node's work is spread over the 32 threads.
//
// A position is held suit by suit. Thread t stands for suit s = t & 3 and seat
// p = (t >> 2) & 3 (the upper half-warp repeats the lower one) and keeps the 13-bit mask
// of the cards seat p holds in suit s; sets of cards (relevant, tried, in play) are kept
// as one 13-bit mask per suit, the same in every thread of that suit. So suit lengths are
// one popcount for all sixteen holdings, playing a card is one masked XOR, a set is one
// 32-bit register, and nothing but the transposition table's key needs 64-bit words. What
// a node does per suit (owner codes, top cards, widening the relevant cards), per table
// way (tags, entries) or per candidate (weights, skipping small cards) runs side by side
// in the threads that stand for it; what is one decision (trick winner, bounds, the next
// move) is the same scalar code in all threads. The stack of frames lies in shared memory.
//
// Decisions, their order and the table's contents are those of ddg_search.cuh (and of the
// reference, src/dd.h:613-939), so node counts per job are equal, node for node; a host
// emulation of the warp (tests/native/warp_replay.cpp) checks it on the CPU.
#pragma once
#include "ddg_search.cuh"

#ifndef DDG_TT_SIG

namespace ddg {

#ifdef __CUDACC__
#define DDG_W __device__ __forceinline__
DDG_W u32 w_ballot(bool p) { return __ballot_sync(0xFFFFFFFFu, p); }
DDG_W u32 w_shfl(u32 v, int src) { return __shfl_sync(0xFFFFFFFFu, v, src); }
DDG_W u32 w_shfl_up1(u32 v) { return __shfl_up_sync(0xFFFFFFFFu, v, 1); }
DDG_W u32 w_or(u32 v) { return __reduce_or_sync(0xFFFFFFFFu, v); }
DDG_W u32 w_max(u32 v) { return __reduce_max_sync(0xFFFFFFFFu, v); }
DDG_W u32 w_min(u32 v) { return __reduce_min_sync(0xFFFFFFFFu, v); }
DDG_W u32 w_add(u32 v) { return __reduce_add_sync(0xFFFFFFFFu, v); }
DDG_W bool w_any(bool p) { return __any_sync(0xFFFFFFFFu, p); }
// The same value in all threads, said so to the compiler: what goes around the search's loops
// passes through this shuffle, and branches on it through a vote, so that it can see that the
// warp stays together. Measured against the same build without them (hard 13-card deals): one
// search alone on an SM 1.35 against 1.17 M nodes/s, every SM full 2.38 against 2.20 G.
DDG_W u32 w_uni(u32 v) { return __shfl_sync(0xFFFFFFFFu, v, 0); }
DDG_W void w_sync() { __syncwarp(); }
DDG_W int w_top(u32 x) { return 31 - __clz((int)x); }   // highest set bit, -1 for 0
DDG_W int w_low(u32 x) { return __ffs((int)x) - 1; }    // lowest set bit, -1 for 0
DDG_W int w_popc(u32 x) { return __popc(x); }
DDG_W u32 w_rev(u32 x) { return __brev(x); }
DDG_W u32 w_shl_hi(u32 hi, u32 lo, int k) { return __funnelshift_l(lo, hi, k); }  // high word of hi:lo << k, k < 32
#else  // the host emulation provides the collectives (warp_emu.hpp)
#define DDG_W static inline
DDG_W bool w_any(bool p) { return w_ballot(p) != 0; }
DDG_W u32 w_uni(u32 v) { return v; }
DDG_W int w_top(u32 x) { return x ? 31 - __builtin_clz(x) : -1; }
DDG_W int w_low(u32 x) { return x ? __builtin_ctz(x) : -1; }
DDG_W int w_popc(u32 x) { return __builtin_popcount(x); }
DDG_W u32 w_shl_hi(u32 hi, u32 lo, int k) { return (u32)(((u64)hi << 32 | lo) << k >> 32); }
DDG_W u32 w_rev(u32 x) {
  u32 r = 0;
  for (int k = 0; k < 32; k++) r |= (x >> k & 1) << (31 - k);
  return r;
}
#endif

// One level of the search in shared memory: what taking its move back needs, and its
// candidates' keys, unordered: the next one is the greatest key below the last one's
// (a key is unique), one reduction over the warp, so the list is never sorted.
struct alignas(16) WarpFrame {
  struct {
    u32 at;     // relevant cards gathered so far | cards tried << 16
    u32 code;   // the rest as it was before this frame's card was played: taking the card back
    u32 cards;  // is loading them. In play at the start of the trick | in a hand << 16
    u32 word;   // of suits 0, 1, 2: state word, w_open_info(), trick
  } suit[4];
  uint16_t m[16];     // cards of every (suit, seat)
  uint16_t keys[16];  // (weight + KEY_BIAS) << 6 | card; 0: no candidate
};
static_assert(sizeof(WarpFrame) == 128, "frames are copied as 16-byte words");
enum { KEY_BIAS = 352 };  // the weights lie within -300 .. 140

// The state word: leader:2 | -:1 | cards played to the trick * 8:2 | -:3 | offset of the
// node's frame:13 | tricks left:4 | tricks NS still need:4.
enum : u32 {
  SW_LEADER = 3, SW_CARD = 8, SW_NP8 = 0x18, SW_FRAME = (u32)sizeof(WarpFrame) << 8, SW_OFF = 0x1FFF00, SW_LEFT = 1u << 21,
  SW_NEED = 1u << 25
};

// Counters, one to a thread.
enum { WCNT_PROBES = 0, WCNT_HITS = 1, WCNT_STORES = 2, WCNT_READS = 3, WCNT_BYTES = 4, WCNT_BOUNDS = 5, WCNT_COUNT = 6 };

// A searcher's job, root search and totals: read and written at root searches only.
struct WarpJob {
  long long job, deal;
  u64 start_nodes, nodes;  // node totals at the job's start / now (flushed)
  u64 total[WCNT_COUNT];   // the threads' counters (flushed)
  u32 jobs_done;
  int8_t strain, decl, last_decl, mode, lo, hi, cards, stage;
};

struct WarpMem {
  WarpFrame fr[STACK_DEPTH];
  u64 hash[14];         // of the trick starts being searched, by tricks left
  // Candidates, handed to threads 0, 1, 2, ... A hand of 13 has at most 13, but device-memory
  // deals come unchecked, and four suits of 13 ranks hold at most 28 runs.
  uint8_t scratch[32];
  WarpJob job;
};

// Registers of a searcher. The same in all threads, unless marked: [s] per suit, [sp] per
// (suit, seat), [t] per thread.
struct WarpState {
  u32 m;      // [sp] cards of the seat in the suit
  u32 all;    // [s] cards in play at the start of the trick
  u32 now;    // [s] cards still in a hand
  u32 code;   // [s] owners of those, two bits each, the highest card's at the top of the word
  u32 rel;    // [s] relevant cards of the node just finished
  u32 at;     // [s] top frame's relevant cards | tried cards << 16
  u32 cnt;    // [t] counter of thread WCNT_*
  u32 st;     // the state word
  u32 trick;  // cards of the trick, a byte each (the bytes from the next one on are 0)
  u32 info;   // top frame's info word
  int trump;
  int leader, nplayed, left, need;  // fields of st, as w_unpack() last read them
  u32 nodes;  // nodes since the last flush
  u32 gen;
#ifdef DDG_BOUNDS_CHECK
  bool fault;  // a bounds check failed
#endif
};
DDG_W void w_unpack(WarpState& w) {
  w.leader = (int)(w.st & SW_LEADER);
  w.nplayed = (int)(w.st >> 3 & 3);
  w.left = (int)(w.st >> 21 & 15);
  w.need = (int)(w.st >> 25 & 15);
}

// Branch weights: what few nodes run is kept out of the line of what most run.
#define W_RARE(x) (__builtin_expect(!!(x), 0))
#define W_OFTEN(x) (__builtin_expect(!!(x), 1))

struct WarpIds {  // what a thread stands for
  int t, s, p;
};

DDG_W void w_count(WarpState& w, const WarpIds& id, int what, u32 k) {
  if (id.t == what) w.cnt += k;
}

// Bounds-checked builds (libddg_check.so): every frame, table bucket, trick hash and candidate
// slot is checked before its access. A check that fails is counted and the access skipped; the
// searcher then ends (w_fault), its job's results unsolved, and the call reports the count as an
// error. (Ways and positions in a bucket are 4-bit fields of 16.) In other builds nothing is left.
#ifdef DDG_BOUNDS_CHECK
DDG_W bool w_in_bounds(WarpState& w, const WarpIds& id, bool ok) {
  if (w_any(!ok)) {
    w_count(w, id, WCNT_BOUNDS, 1);
    w.fault = true;
  }
  return !w_any(!ok);
}
#define W_IN_BOUNDS(ok) w_in_bounds(w, id, ok)
#else
#define W_IN_BOUNDS(ok) true
#endif

// ---- key and owner codes -------------------------------------------------------------------

struct WarpLens {
  u32 hi, lo;  // length_key()
};
// Suit lengths of all hands: one popcount for the 16 holdings, two OR reductions.
DDG_W WarpLens w_lens(const WarpState& w, const WarpIds& id) {
  const u32 part = (u32)w_popc(w.m) << (28 - 4 * (id.t & 7));
  return WarpLens{w_or(id.t & 8 ? 0 : part), w_or(id.t & 8 ? part : 0)};
}
struct WarpKey {
  u32 q, q_hi;  // hash bits 9..40 and 41..47
  u32 bucket, tag;
};
DDG_W WarpKey w_key(const WarpState& w, u64 x, u32 mask) {  // make_key
  WarpKey k;
  k.bucket = (u32)x & mask;
  k.q = (u32)(x >> 9);
  k.q_hi = (u32)(x >> 41) & 0x7Fu;
  k.tag = ((u32)(x >> 32) & 0xFFFF0000u) | ((u32)w.left << 12) | (w.gen << 2) | (u32)w.leader;
  return k;
}

// Owner code of this thread's suit from the hands (a job's start; then w_play keeps it).
DDG_W u32 w_build_code(const WarpState& w, const WarpIds& id) {
  u32 h[4], code = 0;
  for (int q = 0; q < 4; q++) h[q] = w_shfl(w.m, 4 * q + id.s);
  int n = 0;
#pragma unroll
  for (int r = 12; r >= 0; r--) {
    const u32 on = (h[0] | h[1] | h[2] | h[3]) >> r & 1;
    const u32 who = (h[1] >> r & 1) | (h[2] >> r & 1) << 1 | (h[3] >> r & 1) * 3;
    code = on ? code << 2 | who : code;
    n += (int)on;
  }
  return code << 1 << (31 - 2 * n);
}
// The owners of the highest n cards, lowest card in the low bits (n = 0: 0; at most 13).
DDG_W u32 w_pattern(u32 code, int twice_n) { return w_shl_hi(0, code, twice_n); }

// The top n cards of this thread's suit: the suit's eight threads each test two ranks for n
// cards at or above them.
DDG_W u32 w_top_n(const WarpIds& id, u32 all, int n) {
  const int r = id.t >> 2;
  const u32 a = w_ballot(w_popc(all >> r) >= n) >> id.s & 0x11111111u, b = w_ballot(w_popc(all >> (r + 8)) >= n) >> id.s & 0x11111111u;
  const int low = w_popc(a) + w_popc(b) - 1;
  return (all >> low) << low;
}

// A searcher has its table to itself, so its entries are stored as they are (those of tables
// that lanes may share are sealed against torn reads, ddg_tt.cuh).
struct WarpEntry {
  u32 q, w0;     // q: hash bits 9..40 | hash bits 41..47:7 | lb:4 | ub:4 | best:6 | owners 48..57:10, 1 bit free
  u32 w1, own;   // counts:16 | owners 0..15; owners 16..47
};
DDG_W WarpEntry w_entry(const TTBucket* b, int way) {
#ifdef __CUDA_ARCH__
  const uint4 x = *reinterpret_cast<const uint4*>(b->e[way]);
  return WarpEntry{x.x, x.y, x.z, x.w};
#else
  WarpEntry e;
  memcpy(&e, b->e[way], 16);
  return e;
#endif
}
DDG_W void w_entry_put(TTBucket* b, int way, WarpEntry e) {
#ifdef __CUDA_ARCH__
  *reinterpret_cast<uint4*>(b->e[way]) = make_uint4(e.q, e.w0, e.w1, e.own);
#else
  memcpy(b->e[way], &e, 16);
#endif
}

// ---- transposition table -------------------------------------------------------------------

// The probe (tt_probe): thread t looks at tag t & 15; those that match read and check
// their entries side by side. Returns 1, 0 (rel set) or -1 (hint set).
DDG_W int w_probe(WarpState& w, const WarpIds& id, const TTBucket* b, u32 tagw, const WarpKey& k, u32 code, int need,
                  int& hint) {
  hint = -1;
  const bool match = id.t < TT_WAYS && (tagw & ~0xF00u) == k.tag;
  const u32 mm = w_ballot(match);
  w_count(w, id, WCNT_PROBES, 1);
  if (!mm) return -1;
  u32 codes[4];
#pragma unroll
  for (int s = 0; s < 4; s++) codes[s] = w_shfl(code, s);
  bool same = false, decides = false, holds = false;
  int best = 63;
  u32 counts = 0;
  if (match) {
    const WarpEntry e = w_entry(b, (int)((tagw >> 8) & 15));
    counts = e.w1 & 0xFFFFu;
    // Tag, bucket and q are the whole hash of the suit lengths, a bijection, so an entry
    // with this q has these lengths: its counts are no longer than the suits.
    const int b0 = (int)(counts << 1 & 30), b1 = (int)(counts >> 3 & 30), b2 = (int)(counts >> 7 & 30);
    u32 lo = w_pattern(codes[3], (int)(counts >> 11 & 30)), hi = 0;
    hi = w_shl_hi(hi, lo, b2);
    lo = lo << b2 | w_pattern(codes[2], b2);
    hi = w_shl_hi(hi, lo, b1);
    lo = lo << b1 | w_pattern(codes[1], b1);
    hi = w_shl_hi(hi, lo, b0);
    lo = lo << b0 | w_pattern(codes[0], b0);
    same = ((e.q ^ k.q) | ((e.w0 ^ k.q_hi) & 0x7Fu) | (lo ^ (e.w1 >> 16 | e.own << 16)) |
            (hi ^ (e.own >> 16 | (e.w0 >> 21 & 0x3FFu) << 16))) == 0;
    const int lb = (int)(e.w0 >> 7 & 15), ub = (int)(e.w0 >> 11 & 15);
    best = (int)(e.w0 >> 15 & 63);
    holds = lb >= need;
    decides = same && (holds || ub < need);
  }
  const u32 dec = w_ballot(decides), up = w_ballot(decides && holds);
  const u32 before = dec ? (dec & (0u - dec)) - 1 : 0xFFFFu;  // the ways read ahead of the deciding one
  const u32 hints = w_ballot(same && best != 63) & before;
  w_count(w, id, WCNT_READS, (u32)w_popc(mm & (before << 1 | 1)));
  if (dec) {
    const int at = w_low(dec);
    const u32 c = w_shfl(counts, at);
    w.rel = w_top_n(id, w.all, (int)(c >> (4 * id.s)) & 15);
    w_count(w, id, WCNT_HITS, 1);
    return (int)((up >> at) & 1);
  }
  if (W_RARE(hints)) hint = (int)w_shfl((u32)best, w_top(hints));
  return -1;
}

// The store (tt_store) of bounds [lb, ub] for the class of positions that share the
// relevant cards `rel`: each suit's thread makes its owner pattern, each way's thread
// checks its entry, and the tag line shifts by one shuffle.
DDG_W void w_store(WarpState& w, const WarpIds& id, TTBucket* b, u32 tagw, const WarpKey& k, u32 code, u32 rel, int lb,
                   int ub, int best) {
  const u32 above = (u32)w_popc(w.all & (0u - (rel & (0u - rel))));  // cards at or above the lowest relevant one
  const u32 each = w_or(above << (8 * id.s)), upto = each * 0x01010101u;  // a byte a suit; of the suits up to it
  if ((upto >> 24) > MAX_REL) return;
  const u32 n4 = (each | each >> 4) & 0x00FF00FFu, counts = (n4 | n4 >> 8) & 0xFFFFu;
  const int off = 2 * (int)((upto >> (8 * id.s) & 0xFF) - above);
  const u32 pat = w_pattern(code, 2 * (int)above);
  const u32 own_lo = w_or(off < 32 ? pat << off : 0), own_hi = w_or(off < 32 ? w_shl_hi(0, pat, off) : pat << (off & 31));
  WarpEntry e = {k.q, k.q_hi | own_hi >> 16 << 21, counts | own_lo << 16, own_lo >> 16 | own_hi << 16};
  const bool match = id.t < TT_WAYS && (tagw & ~0xF00u) == k.tag;
  const u32 mm = w_ballot(match);
  w_count(w, id, WCNT_STORES, 1);
  bool same = false;
  u32 old = 0;
  if (match) {
    const WarpEntry o = w_entry(b, (int)((tagw >> 8) & 15));
    same = ((o.q ^ e.q) | (o.w1 ^ e.w1) | (o.own ^ e.own) | ((o.w0 ^ e.w0) & ~(0x3FFFu << 7))) == 0;
    old = o.w0 >> 7 & 0x3FFFu;  // lb:4 | ub:4 | best:6
  }
  const u32 sm = w_ballot(same);
  int way;
  if (sm) {  // the class has an entry: the first one is narrowed in place
    const int at = w_low(sm);
    old = w_shfl(old | ((tagw >> 8) & 15) << 16, at);
    way = (int)(old >> 16);
    const int olb = (int)(old & 15), oub = (int)(old >> 4 & 15), obest = (int)(old >> 8 & 63);
    lb = olb > lb ? olb : lb;
    ub = oub < ub ? oub : ub;
    best = best < 0 ? obest : best;
  } else {
    // The way (take_way): the first empty one, else the least 2 * tricks left + age, other
    // generations first; of equal ones the oldest.
    const int age = TT_WAYS - 1 - (id.t & 15);
    const u32 empty = w_ballot(id.t < TT_WAYS && tagw == 0);
    const u32 v = ((tagw >> 2) & 63) != w.gen ? 0 : 1 + 2 * ((tagw >> 12) & 15) + (u32)age;
    const int pos = empty ? TT_WAYS - 1 : TT_WAYS - 1 - (int)(w_min(v << 4 | (u32)age) & 15);
    way = empty ? w_low(empty) : (int)((w_shfl(tagw, pos) >> 8) & 15);
    const u32 prev = w_shfl_up1(tagw);
    if (id.t <= pos) b->tag[id.t] = id.t == 0 ? (k.tag | (u32)way << 8) : prev;
  }
  // (the entries read: up to the one that matches)
  w_count(w, id, WCNT_BYTES, (sm ? 64 + 8 : 64 + 64 + 16) + 16 * (u32)w_popc(mm & ((sm & (0u - sm)) * 2 - 1)));
  e.w0 |= ((u32)lb | (u32)ub << 4 | (u32)(best < 0 ? 63 : best) << 8) << 7;
  if (id.t == TT_WAYS) w_entry_put(b, way, e);
  w_sync();
}

// ---- the top cards of every suit, relative to the leader ------------------------------------

// Per suit, in its threads: lengths of leader, left, partner, right (4 bits each), holders
// of the top three cards relative to the leader (0..3, REL_NONE = no such card; 4 bits
// each from bit 16), and the cards' ranks.
enum { REL_NONE = 4, REL_L = 1, REL_P = 2, REL_R = 3 };
struct WarpTop {
  u32 a, ranks;
};
DDG_W int rt_len(u32 a, int who) { return (int)(a >> (4 * who)) & 15; }
DDG_W int rt_win(u32 a) { return (int)(a >> 16) & 15; }
DDG_W int rt_sec(u32 a) { return (int)(a >> 20) & 15; }
DDG_W int rt_thr(u32 a) { return (int)(a >> 24) & 15; }
DDG_W int rt_rank(u32 r, int k) { return (int)(r >> (4 * k)) & 15; }

DDG_W WarpTop w_make_top(const WarpState& w, const WarpIds& id, const WarpLens& k) {
  const int sh = 12 - 4 * id.s;  // lengths of seats 0..3 in this suit, then rotated to the leader
  const u32 l = ((k.hi >> (sh + 16)) & 15) | ((k.hi >> sh) & 15) << 4 | ((k.lo >> (sh + 16)) & 15) << 8 |
                ((k.lo >> sh) & 15) << 12;
  WarpTop t;
  t.a = ((l | l << 16) >> (4 * w.leader)) & 0xFFFFu;
  // bit 28: of the cards the leader does not hold, partner's is the highest
  const u32 len = (u32)w_popc(w.all);
  const u32 others = (w.code ^ (u32)w.leader * 0x55555555u) & ~(0xFFFFFFFFu >> (2 * len));
  const int pos = (31 - w_top(others)) & 30;
  t.a |= others && ((w.code >> (30 - pos) ^ (u32)w.leader) & 3) == 2 ? 1u << 28 : 0;
  t.ranks = 0;
  u32 a = w.all;
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const u32 c = (u32)w_top(a) & 15;
    const u32 who = a ? ((w.code >> (30 - 2 * j)) - (u32)w.leader) & 3 : (u32)REL_NONE;
    t.ranks |= c << (4 * j);
    t.a |= who << (16 + 4 * j);
    a &= ~(1u << c);
  }
  return t;
}

// ---- QuickTricks and LaterTricks (ddg_bounds.cuh, the same decisions in the same order) ------

struct QtIn {  // one suit as QuickTricks sees it
  int own, lho, part, rho, win, sec, thr;
  u32 ranks;
};
DDG_W QtIn w_qt_in(u32 a, u32 ranks) {
  QtIn q;
  q.own = rt_len(a, 0);
  q.lho = rt_len(a, REL_L);
  q.part = rt_len(a, REL_P);
  q.rho = rt_len(a, REL_R);
  q.win = rt_win(a);
  q.sec = rt_sec(a);
  q.thr = rt_thr(a);
  q.ranks = ranks;
  return q;
}

// One holding side's tricks of a suit whose top card it holds: `a` holds it, `b` is its
// partner (qt_lead_side / qt_lead_plain for the leader, qt_partner_* over the entry).
// side: a side suit of a trump contract. draws: cashing draws the opponents' trumps.
DDG_W int w_qt_suit(const QtIn& c, const WarpIds& id, int suit, bool lead, bool side, bool draws, int cutoff, int& lhoT,
                    int& rhoT, int comm_suit, u32 entry, int qt, u32& wr, int& res) {
  const int a = lead ? c.own : c.part, b = lead ? c.part : c.own;
  const int first = lead ? 0 : REL_P, other = lead ? REL_P : 0;
  const bool out = lhoT == 0 && rhoT == 0;  // both opponents are out of trumps
  const bool clear = !side || out;
  const u32 mine = id.s == suit ? 0xFFFFFFFFu : 0u;
  res = QT_STOP;
  if (!side || ((c.lho != 0 || lhoT == 0) && (c.rho != 0 || rhoT == 0))) {
    wr |= (1u << rt_rank(c.ranks, 0) & mine) | entry;
    if (++qt >= cutoff) return qt;
    if (draws) {
      lhoT = lhoT > 0 ? lhoT - 1 : 0;
      rhoT = rhoT > 0 ? rhoT - 1 : 0;
    }
    if (c.lho <= 1 && c.rho <= 1 && b <= 1 && clear) {
      qt += a - 1;
      if (qt >= cutoff) return qt;
      res = QT_NEXT;
      return qt;
    }
  }
  const bool run = c.sec == first, both = c.sec == other && a > 1 && b > 1;
  if (run || both) {
    if (clear) {
      wr |= (1u << rt_rank(c.ranks, 1) & mine) | (side ? entry : 0);
      if (++qt >= cutoff) return qt;
      if (draws) {
        lhoT = lhoT > 0 ? lhoT - 1 : 0;
        rhoT = rhoT > 0 ? rhoT - 1 : 0;
      }
      if (c.lho <= 2 && c.rho <= 2 && (b <= 2 || (both && a <= 2))) {
        qt += (run || a > b ? a : b) - 2;
        if (qt >= cutoff) return qt;
        res = QT_NEXT;
        return qt;
      }
    }
  } else if (!lead && suit == comm_suit && c.sec == REL_L &&
             (!side || ((c.lho >= 2 || lhoT == 0) && (c.rho >= 2 || rhoT == 0)))) {
    if (c.thr == REL_P) {
      wr |= (1u << rt_rank(c.ranks, 2) & mine) | (side ? entry : 0);
      if (++qt >= cutoff) return qt;
      if (c.own <= 2 && c.lho <= 2 && c.rho <= 2 && clear) {
        qt += c.part - 2;
        if (qt >= cutoff) return qt;
      }
    }
  }
  res = QT_STAY;
  return qt;
}

// Can QuickTricks decide? Every suit's thread bounds its suit's quick tricks from above, as
// if the opponents were out of trumps and partner could be reached; the walk over the
// suits (w_quick_tricks) decides one call in eight, and is left out where the bounds do
// not add up to the cutoff and none of its other answers can come: a suit neither opponent
// holds, a ruff for the one trick needed, no quick trick when the opponents need one.
DDG_W bool w_quick_possible(const WarpState& w, const WarpIds& id, const WarpTop& top, int cutoff, int cutoff_other) {
  const int own = rt_len(top.a, 0), lho = rt_len(top.a, REL_L), part = rt_len(top.a, REL_P), rho = rt_len(top.a, REL_R);
  const int win = rt_win(top.a), sec = rt_sec(top.a), longest = own > part ? own : part;
  const int other = win == 0 ? part : own, most = lho > rho ? lho : rho;
  const bool ours = !(win & 1) && win != REL_NONE;
  // two top cards, or the third behind the left hand's second
  const bool two = (!(sec & 1) && sec != REL_NONE) || (sec == REL_L && rt_thr(top.a) == REL_P);
  const bool lone = (lho | rho) == 0 && longest != 0;
  // Side suits run on only when the opponents' trumps are gone: the leader draws two at most.
  const u32 ta0 = w_shfl(top.a, w.trump & 3), ta = w.trump >= 0 ? ta0 : 0;
  const int drawn = rt_win(ta) == 0 ? 2 : 0;
  const bool clear = w.trump < 0 || id.s == w.trump || (rt_len(ta, REL_L) <= drawn && rt_len(ta, REL_R) <= drawn);
  const bool third = sec == REL_L && rt_thr(top.a) == REL_P;
  const int bound = !clear ? (lone ? 0 : third ? 2 : 1)
                           : lone || (most <= 1 && other <= 1) ? longest : !two ? 1 : most <= 2 ? longest : 2;
  const u32 sum = w_add(id.t < 4 && (ours || lone) ? (u32)bound : 0u);
  return (int)sum >= cutoff || w_any(lone && clear && longest + 1 >= cutoff) || cutoff <= 1 ||
         (cutoff_other <= 1 && (ta & 0xFFFFu) == 0);
}

// QuickTricks (quick_tricks_impl): the leading side's sure tricks against `cutoff`;
// decided = the answer is known (a count > 0: the leading side makes it).
DDG_W int w_quick_tricks(const WarpState& w, const WarpIds& id, const WarpTop& top, int cutoff, int cutoff_other, u32& wr,
                         bool& decided) {
  const int trump = w.trump;
  wr = 0;
  decided = true;
  const bool has_t = trump >= 0;
  const u32 ta = has_t ? w_shfl(top.a, trump) : 0;
  const int tl = rt_len(ta, REL_L), tr = rt_len(ta, REL_R);
  // The entry to partner: every suit's thread tests its suit, the first in order is taken.
  const bool safe = !has_t || ((rt_len(top.a, REL_L) != 0 || tl == 0) && (rt_len(top.a, REL_R) != 0 || tr == 0));
  const bool by_win = rt_win(top.a) == REL_P && rt_len(top.a, 0) != 0;
  const bool by_sec = rt_sec(top.a) == REL_P && rt_win(top.a) == 0 && rt_len(top.a, 0) >= 2 && rt_len(top.a, REL_P) >= 2;
  const u32 entries = w_ballot(id.t < 4 && id.s != trump && safe && (by_win || by_sec));
  int comm_suit = w_low(entries);
  if (comm_suit < 0 && has_t && rt_len(ta, 0) != 0 && rt_win(ta) == REL_P) comm_suit = trump;
  const bool comm = comm_suit >= 0;
  u32 entry = 0;  // [s] the entry card
  if (id.s == comm_suit) entry = 1u << rt_rank(top.ranks, by_win ? 0 : 1);
  // in the trump suit the entry is partner's top card, which by_win says as well
  // The loop's state in one word: suit:3 | ruffed:1 | the opponents' trumps:4, 4 | count.
  u32 state = (u32)(has_t ? trump : 0) | (u32)tl << 4 | (u32)tr << 8;
  for (;;) {
    state = w_uni(state);
    const int suit = (int)(state & 7);
    if (suit > 3) break;
    u32 ruffed = state & 8;
    int lhoT = (int)(state >> 4 & 15), rhoT = (int)(state >> 8 & 15), qt = (int)(state >> 12);
    const QtIn c = w_qt_in(w_shfl(top.a, suit), w_shfl(top.ranks, suit));
    const bool side = has_t && trump != suit;
    const bool no_ruff = !side || (lhoT == 0 && rhoT == 0);
    bool one_hand = false;
    if ((c.lho | c.rho) == 0) {
      const bool only_lead = c.part == 0, only_part = comm && c.own == 0 && !only_lead;
      one_hand = only_lead || only_part;
      if (!only_lead) {
        // The sure length of the partnership's suit may decide at once (qt_blocked_sum, from
        // the leader's side and, with an entry, from partner's).
        const bool in_t = has_t && suit == trump;
        const int more = c.own > c.part ? c.own : c.part, less = c.own < c.part ? c.own : c.part;
        const bool l0 = rt_len(top.a, 0) != 0, l2 = rt_len(top.a, REL_P) != 0;
        const bool by_lead = w_any(id.s != trump && l0 && !l2) && c.own >= c.part;
        const bool by_part = w_any(id.s != trump && !l0 && l2) && c.own <= c.part;
        const int sum1 = in_t ? more + by_lead : less, sum2 = in_t ? more + by_part : less;
        if (no_ruff && sum1 >= cutoff) return sum1;
        if (comm && !only_part && no_ruff && sum2 >= cutoff) {
          if (in_t) wr |= entry;
          return sum2;
        }
      }
      if (one_hand && no_ruff) {  // its cards (partner's over the entry)
        qt += only_lead ? c.own : c.part;
        if (only_part) wr |= entry;
        if (qt >= cutoff) return qt;
      }
    }
    if (!one_hand && c.win != REL_NONE) {
      int res = QT_STAY;
      if (c.win == 0 || (c.win == REL_P && comm)) {
        const bool lead = c.win == 0, draws = lead && has_t && trump == suit && suit != comm_suit;
        qt = w_qt_suit(c, id, suit, lead, side, draws, cutoff, lhoT, rhoT, comm_suit, lead ? 0u : entry, qt, wr, res);
        if (res == QT_STOP) return qt;
      }
      // A ruff by partner.
      if (res == QT_STAY && side && c.own > 0 && !ruffed && c.part == 0 && rt_len(ta, REL_P) > 0 &&
          (qt == 0 || (c.win != 0 && c.win != REL_P && rt_win(ta) != 0 && rt_win(ta) != REL_P))) {
        if ((c.rho > 0 || tr == 0) && (c.lho > 0 || tl == 0)) {
          ruffed = 8;  // nobody can overruff
          if (1 >= cutoff) return 1;
        } else {
          const u32 pt = w_shfl(w.m, 4 * ((w.leader + 2) & 3) + trump);
          const u32 lt = w_shfl(w.m, 4 * ((w.leader + 1) & 3) + trump);
          const u32 rt = w_shfl(w.m, 4 * ((w.leader + 3) & 3) + trump);
          if (((c.lho == 0 ? lt : 0) | (c.rho == 0 ? rt : 0)) < pt) {
            ruffed = 8;
            if (id.s == trump) wr |= 1u << w_top(pt);
            if (1 >= cutoff) return 1;
          }
        }
      }
    }
    state = (u32)qt_next_suit(suit, trump) | ruffed | (u32)lhoT << 4 | (u32)rhoT << 8 | (u32)qt << 12;
  }
  const int qt = (int)(state >> 12);
  if (qt == 0 && (!has_t || rt_win(ta) == REL_NONE)) {
    // No quick trick: the opponents win the first trick with a top card.
    if (rt_win(top.a) != REL_NONE && rt_len(top.a, 0) > 0) wr = 1u << rt_rank(top.ranks, 0);
    if (1 >= cutoff_other) return 0;
  }
  decided = false;
  return qt;
}

// LaterTricks (later_min_impl / later_max_impl): true when the bound decides the node (NS
// fail when NS lead, NS make it when EW lead). Written for the leader's side: the other
// side takes at least one trick later.
DDG_W bool w_later_tricks(const WarpState& w, const WarpIds& id, const WarpTop& top, u32& wr) {
  const bool ns = ns_side(w.leader);
  const int dq = w.left - 1, need = w.need;
  wr = 0;
  const u32 ta = w.trump >= 0 ? w_shfl(top.a, w.trump) : 0;
  const bool nt = w.trump < 0 || rt_win(ta) == REL_NONE;
  if (nt) {
    // Tricks the leader's side can take with its own top cards' suits.
    const int win = rt_win(top.a);
    const bool ours = win == 0 || win == REL_P;
    const int l0 = rt_len(top.a, 0), l1 = rt_len(top.a, 1), l2 = rt_len(top.a, 2), l3 = rt_len(top.a, 3);
    const int pair = l0 > l2 ? l0 : l2;
    const int sum = (int)w_add(id.t < 4 && ours ? (u32)pair : 0u);
    if (sum <= 0) return false;
    if (ns) {
      if (!(sum < need) || dq >= need) return false;
    } else {
      if (!(dq + 1 - sum >= need) || 1 < need) return false;
    }
    const bool theirs = win == 1 || win == 3;  // a top card of the other side with another hand in the suit
    const bool others = win == 1 ? (l0 | l2 | l3) != 0 : (l0 | l1 | l2) != 0;
    if (theirs && others) wr = 1u << rt_rank(top.ranks, 0);
    return true;
  }
  // With trumps about, all but one answer needs the bound within two tricks of an end.
  const bool near = ns ? need >= w.left - 1 : need <= 2;
  if (!near && (rt_len(ta, 0) | rt_len(ta, REL_P)) != 0) return false;
  const u32 tk = w_shfl(top.ranks, w.trump);
  const int win = rt_win(ta), sec = rt_sec(ta), thr = rt_thr(ta);
  const bool win_ours = win == 0 || win == REL_P;
  const u32 at_trump = id.s == w.trump ? 0xFFFFFFFFu : 0u;
  // ns: "not even dq tricks are enough"; ew: "one trick is enough"
  const bool one = ns ? dq < need : 1 >= need;
  if (!win_ours) {
    if (rt_len(ta, 0) == 0 && rt_len(ta, REL_P) == 0) {
      const int a = rt_len(ta, REL_L), b = rt_len(ta, REL_R);
      const int m = a > b ? a : b;
      return ns ? dq + 1 - m < need : m >= need;
    }
    if (one) {
      wr = 1u << rt_rank(tk, 0) & at_trump;
      return true;
    }
    if (ns ? dq == need : 2 >= need) {
      if (sec == REL_NONE) return false;
      const bool sec_theirs = sec == 1 || sec == 3;
      if (sec_theirs && (rt_len(ta, 1) > 1 || rt_len(ta, 3) > 1)) {
        wr = 1u << rt_rank(tk, 1) & at_trump;
        return true;
      }
    }
    return false;
  }
  if (sec == REL_NONE || sec == 0 || sec == REL_P || rt_len(ta, sec) <= 1) return false;
  if (win == ((sec + 3) & 3)) {
    if (one) {
      wr = 1u << rt_rank(tk, 1) & at_trump;
      return true;
    }
  } else {
    if (thr == REL_NONE) return false;
    if ((thr == 1 || thr == 3) && one) {
      wr = 1u << rt_rank(tk, 2) & at_trump;
      return true;
    }
  }
  return false;
}

// The second hand's QuickTricks (quick_tricks_2nd_impl). Neither it nor its partner has
// played to the trick, so "holds the suit's top card at the trick's start" is a test of
// its cards.
DDG_W bool w_quick_2nd(const WarpState& w, const WarpIds& id, u32& wr) {
  const int lead = (int)(w.trick & 0xFF), ls = card_suit(lead), trump = w.trump;
  const int hand = lho_of(w.leader), P = partner_of(hand), third = lho_of(hand);
  const int cutoff = ns_side(hand) ? w.need : w.left - w.need + 1;
  wr = 0;
  if (trump >= 0 && cutoff > 1) return false;  // with trumps it counts this trick only
  const u32 me = w_shfl(w.m, 4 * hand + ls), pd = w_shfl(w.m, 4 * P + ls), th = w_shfl(w.m, 4 * third + ls);
  const u32 ranks = me | pd, bit = 1u << (lead & 15);
  const bool wins = ranks > (bit | th);
  bool by_rank = true;
  if (trump >= 0 && ls != trump) {
    const u32 T = w_ballot(id.s == trump && w.m != 0);  // seats that hold a trump: bits 4 * seat + trump
    const bool we_ruff = (!me && (T >> (4 * hand + trump) & 1)) || (!pd && (T >> (4 * P + trump) & 1));
    const bool they_ruff = !th && (T >> (4 * third + trump) & 1);
    if (they_ruff) return false;
    by_rank = !we_ruff;
  }
  if (by_rank && !wins) return false;
  if (by_rank && id.s == ls) wr = 1u << w_top(ranks);
  if (1 >= cutoff) return true;
  const int hh = me > pd ? hand : P;
  const u32 mine = w_shfl(w.m, 4 * hh + id.s);
  const int c1 = w_top(w.all);
  const int c2 = w_top(w.all & ~(c1 >= 0 ? 1u << c1 : 0u));
  const bool has1 = c1 >= 0 && (mine >> c1 & 1);
  const bool has2 = c2 >= 0 && (mine >> c2 & 1);
  int q = 1;
  const u32 top2 = w_ballot(id.t < 4 && id.s == ls && has1 && has2);
  if (top2) {
    q++;
    if (id.s == ls) wr |= 1u << c2;
    if (q >= cutoff) return true;
  }
  // The other suits in order, each adding its tricks; the cards of those up to the one
  // that reaches the cutoff count.
  const bool lone = mine != 0 && !(w.now & ~mine);  // nobody else holds the suit
  const int inc = id.s == ls || !mine ? 0 : lone ? w_popc(mine) : has1 ? 1 : 0;
  const u32 upto = w_or((u32)inc << (4 * id.s)) * 0x1111u >> (4 * id.s) & 15;  // (at most 13 in all)
  const u32 reached = w_ballot(id.t < 4 && q + (int)upto >= cutoff);
  if (!reached) return false;
  const int until = w_low(reached);
  if (inc && !lone && id.s <= until) wr |= 1u << c1;
  return true;
}

// ---- move generation -----------------------------------------------------------------------

// Cards of a holding that are the top of their run (run_tops for one suit). With the highest
// rank in the lowest bit, a run is a stretch of ones in (own or not in play); adding own
// sends a carry from its first own card through the rest, which leaves there a zero at the
// first own card and a one at every later one.
DDG_W u32 w_run_tops(u32 own, u32 all) {
  const u32 o = w_rev(own);
  return w_rev(o & ~(w_rev(own | ~all) + o));
}
// Is the highest card of `cards` one of `mine`? (Sets compare like their highest cards.)
DDG_W bool w_top_is(u32 cards, u32 mine) { return (cards & mine) > (cards & ~mine); }

// The DDS lead weight (lead_weight) of `card` in this thread; top, hands and lengths of the
// card's suit come from its threads.
DDG_W int w_lead_weight(const WarpState& w, const WarpTop& top, int card, int hint) {
  const int s = card_suit(card), r = card & 15, lead = w.leader, trump = w.trump;
  const u32 a = w_shfl(top.a, s), tk = w_shfl(top.ranks, s), all = w_shfl(w.all, s);
  const u32 own = w_shfl(w.m, 4 * lead + s);
  u32 ta = 0, hLT = 0, hPT = 0, hRT = 0;
  if (trump >= 0) {
    ta = w_shfl(top.a, trump);
    hLT = w_shfl(w.m, 4 * lho_of(lead) + trump);
    hPT = w_shfl(w.m, 4 * partner_of(lead) + trump);
    hRT = w_shfl(w.m, 4 * rho_of(lead) + trump);
  }
  const u32 bit = 1u << r;
  bool tt = false;  // the card, or one alike, is the hint
  if (hint >= 0 && card_suit(hint) == s) {
    const int hr = hint & 15, lo = r < hr ? r : hr, hi = r < hr ? hr : r;
    const u32 between = ((1u << hi) - 1) & ~((2u << lo) - 1);
    tt = (all & ~own & between) == 0;
  }
  const int r_rank = w_popc(all >> r);
  const bool seq = w_top_is(all & (bit - 1), own);  // the next card down is the leader's too
  const int lenL = rt_len(a, REL_L), lenR = rt_len(a, REL_R), lenP = rt_len(a, REL_P);
  const u32 cnt = (u32)((lenL == 0 ? w.left : lenL) + (lenR == 0 ? w.left : lenR)) << 2;
  const int w1 = rt_win(a), w2 = rt_sec(a), w3 = rt_thr(a);
  const bool is_win = rt_rank(tk, 0) == r, is_sec = w2 != REL_NONE && rt_rank(tk, 1) == r;
  const bool drop = (lenL == 1 && w1 == REL_L) || (lenR == 1 && w1 == REL_R);
  const bool p_long = (w2 == 0 && w3 == REL_P && lenP > 1) || (w2 == REL_P && w3 == 0 && lenP > 1);
  const bool pp = w2 == REL_P && w3 == REL_P;
  const bool w1_0 = w1 == 0, w1_p = w1 == REL_P, w2_p = w2 == REL_P;
  const bool tops = (a >> 28 & 1) != 0, lead_sec = seq & is_sec;
  int delta, base;
  bool with_rank;  // weight = delta + base (+ r_rank)
  if (trump >= 0 && rt_win(ta) != REL_NONE) {
    const int tP = rt_len(ta, REL_P);
    const bool side = s != trump;
    const bool ruffL = (lenL == 0) & (rt_len(ta, REL_L) != 0), ruffR = (lenR == 0) & (rt_len(ta, REL_R) != 0);
    const u32 over = (ruffL ? hLT : 0) | (ruffR ? hRT : 0);  // trumps of the opponents that can ruff
    const bool p_ruffs = (lenP == 0) & (tP != 0);
    delta = -(int)((cnt << 5) / 13);
    delta += side & (ruffL | ruffR) ? -12 : 0;
    delta += side & p_ruffs & (lenR > 0) ? 17 : 0;
    delta += (w1 == REL_R) | (w2 == REL_R) ? (lenR != 1 ? -12 : 0) : (w1 == REL_L) & w2_p & (lenP != 1) ? 27 : 0;
    delta += side & (rt_len(a, 0) == 1) & (rt_len(ta, 0) > 0) & (lenP > 1) & w1_p ? 19 : 0;
    const bool ruff_wins = hPT > over;
    const bool win = is_win | tops ? !side | (is_win & p_ruffs ? ruff_wins : over == 0) : side & p_ruffs & ruff_wins;
    if (win) {
      base = drop ? 35 : w1_0 ? (w2_p ? 48 : is_win ? 31 : -3) : w1_p ? (w2 == 0 ? 42 : 28) : lead_sec ? 40 : seq ? 22 : 11;
      with_rank = drop | (w1_0 ? w2_p | !is_win : w1_p | !lead_sec);
      base += tt ? 18 : 0;
    } else {
      delta += pp ? 20 : p_long ? 13 : 0;
      base = drop ? 2 : w1_0 ? (w2_p ? 33 : is_win ? 38 : -14) : w1_p ? 34 : lead_sec ? 35 : 15 - r;
      with_rank = drop | (w1_0 ? w2_p | !is_win : w1_p);
    }
    return delta + base + (with_rank ? r_rank : 0);
  }
  delta = -(int)((cnt << 5) / 19) - (lenP == 0 ? 9 : 0);
  if (is_win | tops) {
    const bool safe = ((w2 != REL_L) | (lenL == 1)) & ((w2 != REL_R) | (lenR == 1));
    delta += w2 == REL_R ? (lenR != 1 ? -1 : 0) : w2 == REL_L ? (lenL != 1 ? 22 : 16) : 0;
    return delta + (safe ? 45 : 18) + (tt ? 32 : 0) + r_rank;
  }
  delta += (w1 == REL_R) | (w2 == REL_R) ? (lenR != 1 ? -10 : 0) : (w1 == REL_L) & w2_p & (lenP != 1) ? 31 : 0;
  delta += pp ? 35 : p_long ? 25 : 0;
  base = drop ? 28 : w1_0 ? -17 : !seq ? 12 : is_sec ? 48 : 29;
  const int by = drop | w1_0 | !seq ? r_rank : is_sec ? 0 : -r_rank;
  return delta + base + by + (tt ? 19 : 0);
}

// The DDS follow weights (follow_weight) of `card` in this thread; n = cards played. What
// is the same for all candidates of a node is decided once (the branches); what differs
// from card to card is chosen by selects, so the warp does not diverge.
DDG_W int w_follow_weight(const WarpState& w, int n, int seat, bool is_void, int card) {
  const int lead = w.leader, trump = w.trump;
  const bool has_t = trump >= 0;
  const int c0 = (int)(w.trick & 0xFF), ls = card_suit(c0);
  const int s = card_suit(card), r = card & 15, rank = r + 2;
  const int P = partner_of(lead), R = rho_of(lead);
  const u32 hRL = w_shfl(w.m, 4 * R + ls), hRT0 = w_shfl(w.m, 4 * R + (trump & 3)), hRT = has_t ? hRT0 : 0;
  const u32 all = w_shfl(w.all, s), now = w_shfl(w.now, s), me = w_shfl(w.m, 4 * seat + s);
  const int r_rank = w_popc(now >> r);
  const u32 bit = 1u << r, lead_bit = 1u << (c0 & 15);
  const int c1 = (int)(w.trick >> 8 & 0xFF), c2 = (int)(w.trick >> 16 & 0xFF);
  const int high1 = n > 1 && beats(c1, c0, trump) ? 1 : 0, move1 = high1 ? c1 : c0;
  // Cards of one suit compare as their bits do, and a card with a hand's highest as its bit
  // with the hand's set.
  if (!is_void) {  // the 2nd hand (the others' order: w_follow_floor)
    const u32 hPL = w_shfl(w.m, 4 * P + ls), hPT0 = w_shfl(w.m, 4 * P + (trump & 3)), hPT = has_t ? hPT0 : 0;
    const u32 hLL = w_shfl(w.m, 4 * lead + ls);
    const bool seq = w_top_is(all & (bit - 1), me);
    const bool over = bit > (hPL | lead_bit), pd_over = hRL > (hPL | lead_bit), above = bit > lead_bit;
    const bool under3 = (hPL != 0) & ((hPL & (bit - 1)) == 0);  // below all of the third hand's
    const bool under = under3 | ((hRL != 0) & ((hRL & (bit - 1)) == 0));
    int base;
    bool by_rank;  // weight = base - rank, else base + r_rank
    if (has_t) {
      const bool side = ls != trump, pd_ruffs = !hRL && hRT;
      const bool p_follows = hPL || !hPT, pd_over_ruffs = hRT > hPT;
      const bool u1 = !side || p_follows || (pd_ruffs && pd_over_ruffs), u2 = !side || p_follows;
      const bool u3 = side && pd_ruffs && (p_follows || pd_over_ruffs), u4 = side && pd_ruffs;
      const bool lead_high = lead_bit > (hPL | hRL);
      const bool win = over ? u1 : pd_over ? u2 : lead_high & !above ? u3 : u4;
      const bool keep = hRL > lead_bit && hLL > hRL;
      const int high = bit < hRL ? 78 : bit > hPL ? 73 : seq ? 62 : 49;
      const int on_win = under3 ? 40 : keep ? 41 : above ? high : hRL ? 47 : 40;
      const int on_loss = under ? -9 : !above ? -16 : seq ? 22 : 10;
      base = win ? on_win : on_loss;
      by_rank = win ? !(under3 | keep) : !(under | !above);
    } else {
      base = pd_over ? 0 : over ? 81 : under ? -3 : !above ? -11 : seq ? 10 : 13;
      by_rank = pd_over | over | !(under | !above | seq);
    }
    return base + (by_rank ? -rank : r_rank);
  }
  // Void in the led suit: weight = base - rank (or + r_rank) + the length's share (64 * length
  // / D, by a multiplication) - a penalty for a bare top card or a guarded second one.
  enum : u32 { K23 = 182361, K24 = 174763, K27 = 155344, K33 = 127100, K36 = 116509, K40 = 104858, K44 = 95326, K50 = 83886 };
  const u32 length = (u32)w_popc(me);
  const int t1 = w_top(all) & 31, t2 = w_top(all & ~(1u << t1));
  const bool one = (length == 1) & (me >> t1 & 1), two = (length == 2) & (t2 >= 0) & (me >> (t2 & 31) & 1);
  const bool ruff = s == trump;
  int base = 0, pen2 = 0, pen1 = 0;
  u32 K;
  bool with_rank = false;
  if (n == 1) {
    const u32 hPL = w_shfl(w.m, 4 * P + ls), hPT0 = w_shfl(w.m, 4 * P + (trump & 3)), hPT = has_t ? hPT0 : 0;
    const bool r_over = hRL > (hPL | lead_bit);  // 4th hand beats the trick
    K = r_over ? K23 : K33;
    pen2 = r_over ? 2 : 6;
    pen1 = r_over ? 3 : 8;
    if (has_t) {
      const bool p_in = hPL != 0, r_ruffs = !hRL && hRT;
      const bool pd_wins = p_in ? r_over || r_ruffs : (!hRL && hRT > hPT) || (!hPT && hRL > lead_bit);
      const bool safe = p_in || (r_ruffs && hRT > hPT);
      const bool high = ls == trump ? r_over : ruff ? safe | (bit > hPT) : pd_wins;
      base = ls == trump ? 0 : ruff ? (high ? 24 : 15) : (high ? 60 : -2);
      K = high ? K44 : K36;
      pen2 = high ? 0 : 4;
      pen1 = 0;
    }
  } else if (n == 2) {
    K = K24;
    pen2 = pen1 = 4;
    if (has_t) {
      const int m1r = rank2(move1);
      const u32 hLL = w_shfl(w.m, 4 * lead + ls), allL = w_shfl(w.all, ls);
      // the second card of the led suit was the leader's at the trick's start
      const int l2 = w_top(allL & ~(1u << (w_top(allL) & 31)));
      const bool sec_lead = l2 >= 0 && ((hLL | lead_bit) >> (l2 & 31) & 1);
      const bool covered = high1 == 0 && lead_bit > hRL && (hRL || !hRT);
      const int follows = high1 == 0 ? (sec_lead ? 36 : 48) : 72, ruffed = high1 == 0 ? -12 : 36;
      const bool ruffing = ruff & (ls != trump), under = (card_suit(move1) == trump) & (rank < m1r);
      base = !ruffing ? 0 : covered ? -50 : under ? -32 : hRL ? follows : bit > hRT ? 48 : ruffed;
      K = ruffing ? (covered ? 0 : under ? K40 : K50) : K40;
      with_rank = ruffing & !covered & under;
      pen2 = pen1 = 0;
    }
  } else {
    const bool h2 = beats(c2, move1, trump);
    const int move2 = h2 ? c2 : move1;
    K = has_t ? K24 : K27;
    pen2 = has_t ? 2 : 6;
    pen1 = has_t ? 0 : 8;
    if (has_t && ls != trump) {
      const bool ours = !h2 && high1;  // partner is winning
      const bool under = (card_suit(move2) == trump) & (rank <= rank2(move2));
      base = ours ? (ruff ? 2 : 25) : ruff ? (under ? -13 : 33) : 14;
      with_rank = ruff & !ours;
      K = with_rank ? 0 : K;
      pen2 = with_rank ? 0 : pen2;
    }
  }
  return base + (with_rank ? r_rank : -rank) + (int)(length * K >> 16) - (two ? pen2 : one ? pen1 : 0);
}

// The 3rd or 4th hand follows suit: the DDS weight is up - rank for a card that wins and
// -rank for one that does not, with `up` above any rank and "wins" a threshold, so the order
// is the winners from the lowest up, then the others from the lowest up. Returns the set
// that a winner's bit exceeds (all ones: no card wins).
DDG_W u32 w_follow_floor(const WarpState& w, int n, int seat) {
  const int trump = w.trump, c0 = (int)(w.trick & 0xFF), c1 = (int)(w.trick >> 8 & 0xFF), ls = card_suit(c0);
  const bool high1 = beats(c1, c0, trump);
  const int move1 = high1 ? c1 : c0;
  const bool side = trump >= 0 && ls != trump;
  const u32 none = 0xFFFFFFFFu;
  if (n == 3) {
    const int c2 = (int)(w.trick >> 16 & 0xFF);
    const bool h2 = beats(c2, move1, trump);
    const int move2 = h2 ? c2 : move1;
    return (!h2 && high1) || (side && card_suit(move2) == trump) ? none : 1u << (move2 & 15);
  }
  const u32 fourth = w_shfl(w.m, 4 * rho_of(w.leader) + ls), third = w_shfl(w.m, 4 * seat + ls);
  const u32 b1 = 1u << (move1 & 15), lead_bit = 1u << (c0 & 15);
  if (side && card_suit(move1) == trump) return none;
  if (side && high1 && !fourth) return b1;
  if (!high1 && (lead_bit > fourth || (side && !fourth))) return none;
  if ((fourth && third < (fourth & (0u - fourth))) || third < b1) return none;
  if (trump >= 0 && third > fourth) return ls == trump || high1 ? fourth | b1 : fourth;
  return trump >= 0 && ls == trump ? none : fourth | b1;
}

// Hands the cards of `cm` ([sp], the threads of `seat`) to threads 0, 1, 2, ...: thread
// t looks at cards t and t + 32. Returns their number; `card` is this thread's.
DDG_W int w_compact(WarpState& w, const WarpIds& id, WarpMem& sm, u32 cm, int seat, int& card) {
  const u32 a = w_shfl(cm, 4 * seat + (id.t >> 4)), b = w_shfl(cm, 4 * seat + 2 + (id.t >> 4));
  const bool ha = a >> (id.t & 15) & 1, hb = b >> (id.t & 15) & 1;
  const u32 ma = w_ballot(ha), mb = w_ballot(hb), lt = (1u << id.t) - 1;
  if (!W_IN_BOUNDS(w_popc(ma) + w_popc(mb) <= 13)) return 0;
  if (ha) sm.scratch[w_popc(ma & lt)] = (uint8_t)id.t;
  if (hb) sm.scratch[w_popc(ma) + w_popc(mb & lt)] = (uint8_t)(id.t + 32);
  w_sync();
  card = sm.scratch[id.t & 15] & 63;
  const int n = w_popc(ma) + w_popc(mb);
  w_sync();
  return n;
}

// The frame's info word: value when no child cuts:1 | seat:2 | more than one candidate:1 | key
// of the one being searched:15 | win card:7 (64 = none; set when it completed a trick).
DDG_W u32 w_open_info(int seat, bool more) { return (u32)(!ns_side(seat)) | (u32)seat << 1 | (u32)more << 3; }
DDG_W int wi_result(u32 info) { return (int)(info & 1); }
DDG_W int wi_seat(u32 info) { return (int)(info >> 1) & 3; }
DDG_W bool wi_more(u32 info) { return info >> 3 & 1; }
DDG_W u32 wi_key(u32 info) { return info >> 4 & 0x7FFFu; }
DDG_W int wi_win_card(u32 info) { return (int)(info >> 19) & 127; }
DDG_W int key_card(u32 key) { return (int)(key & 63); }
enum : u32 { WI_KEEP = 15 };  // what a play leaves

DDG_W u32 w_tags(const TTBucket* b, const WarpIds& id) { return b->tag[id.t & 15]; }

// ENTER at a trick start (enter_lead): cutoffs, the last trick, the TT probe, the bounds. The
// value (w.rel set; `store`: a bound's, to be stored), or -1 when the node expands.
template <class Env>
DDG_W int w_lead(WarpState& w, const WarpIds& id, WarpMem& sm, Env& env, bool& store, WarpTop& top, int& hint) {
  w.rel = 0;
  if (w.need <= 0) return 1;
  if (w.left < w.need) return 0;
  if (W_RARE(w.left == 1)) {
    const u32 bt = w_ballot(id.s == w.trump && w.all != 0);
    const int su = bt ? w.trump : w_low(w_ballot(id.p == w.leader && w.m != 0)) & 3;
    const u32 in = w_shfl(w.all, su);
    if (id.s == su && w_popc(in) >= 2) w.rel = 1u << w_top(in);
    return (int)(~w_shfl(w.code, su) >> 30 & 1);  // the top card's holder is N or S
  }
  const WarpLens lens = w_lens(w, id);
  const u64 x = key_hash((u64)lens.hi << 32 | lens.lo, w.leader);
  const WarpKey k = w_key(w, x, env.mask());
  if (!W_IN_BOUNDS(k.bucket <= env.mask() && w.left < 14)) return 0;
  const TTBucket* b = env.table() + k.bucket;
  const int hit = w_probe(w, id, b, w_tags(b, id), k, w.code, w.need, hint);
  if (W_OFTEN(hit >= 0)) return hit;
  if (id.t == 0) sm.hash[w.left] = x;  // for the store
  w_sync();
  top = w_make_top(w, id, lens);
  const bool ns_lead = ns_side(w.leader);
  const int cut_ns = w.need, cut_ew = w.left - w.need + 1;
  bool decided;
  u32 wr;
  int q = 0, v;
  const int cut = ns_lead ? cut_ns : cut_ew, cut_other = ns_lead ? cut_ew : cut_ns;
  decided = w_quick_possible(w, id, top, cut, cut_other);
  if (W_RARE(decided)) q = w_quick_tricks(w, id, top, cut, cut_other, wr, decided);
  if (decided) v = ns_lead ? q != 0 : q == 0;
  else if (w_later_tricks(w, id, top, wr)) v = !ns_lead;
  else return -1;
  w.rel = wr;
  store = true;
  return v;
}

// A trick start's result goes to the table (a bound's, or a finished node's with its
// cutting card `best` or -1).
template <class Env>
DDG_W void w_put(WarpState& w, const WarpIds& id, const WarpMem& sm, Env& env, int v, int best) {
  if (!W_IN_BOUNDS(w.left < 14)) return;
  const WarpKey k = w_key(w, sm.hash[w.left], env.mask());
  if (!W_IN_BOUNDS(k.bucket <= env.mask())) return;
  TTBucket* b = env.table() + k.bucket;
  w_store(w, id, b, w_tags(b, id), k, w.code, w.rel, v ? w.need : 0, v ? w.left : w.need - 1, best);
}

DDG_W WarpFrame& w_frame(WarpMem& sm, u32 st) {
  return *reinterpret_cast<WarpFrame*>(reinterpret_cast<char*>(sm.fr) + (st >> 8 & 0x1FFF));
}

// A node expands (gen_moves_lead, gen_moves_follow): its candidates, one per run of alike
// cards, with their DDS weights, into a fresh frame. Returns the first one's key.
template <class Env>
DDG_W u32 w_expand(WarpState& w, const WarpIds& id, WarpMem& sm, Env& env, const WarpTop& top, int hint) {
  const int seat = (w.leader + w.nplayed) & 3, ls = (int)(w.trick >> 4) & 3;
  const u32 cm = w_run_tops(w.m, w.all);
  const u32 in_led = w_shfl(cm, 4 * seat + ls);
  const u32 led = w.nplayed ? in_led : 0;
  u32 who = led;  // the threads that stand for a candidate
  int n = w_popc(led), card = ls * 16 + (id.t & 15);  // following suit: thread r for rank r
  if (!led) {
    n = w_compact(w, id, sm, cm, seat, card);
    who = (1u << n) - 1;
  }
  w.at = 0;
  w.info = w_open_info(seat, n != 1);
  if (n == 1) return 64 | w_shfl((u32)card, w_low(who));
  int weight;
  if (W_RARE(w.nplayed == 0)) {
    if (hint < 0 && (w.st & SW_OFF) == 0) {  // the root, no TT move: an outside hint, when the leader holds it
      const int h = env.root_hint(sm.job);
      if (h >= 0 && h < 64 && (w_shfl(w.m, 4 * seat + (h >> 4)) >> (h & 15) & 1)) hint = h;
    }
    weight = w_lead_weight(w, top, card, hint);
  } else if (led && w.nplayed > 1) {
    weight = ((1u << (card & 15)) > w_follow_floor(w, w.nplayed, seat) ? 16 : 0) - (card & 15);
  } else {
    weight = w_follow_weight(w, w.nplayed, seat, !led, card);
  }
  const u32 key = who >> id.t & 1 ? (u32)(weight + KEY_BIAS) << 6 | (u32)card : 0;
  if (!W_IN_BOUNDS((w.st & SW_OFF) < STACK_DEPTH * SW_FRAME)) return 0;
  if (id.t < 16) w_frame(sm, w.st).keys[id.t] = (uint16_t)key;
  return w_max(key);
}

// ENTER inside a trick (enter_follow): the second hand's QuickTricks.
DDG_W int w_enter_follow(WarpState& w, const WarpIds& id) {
  if (w.nplayed != 1) return -1;
  u32 wr;
  if (!w_quick_2nd(w, id, wr)) return -1;
  w.rel = wr;
  return ns_side(lho_of(w.leader)) ? 1 : 0;
}

// Plays the card of `key` from the top frame and pushes the frame (play): at the fourth card the
// trick is settled and the frame keeps what taking it back needs.
DDG_W void w_play(WarpState& w, const WarpIds& id, WarpMem& sm, u32 key) {
  if (!W_IN_BOUNDS((w.st & SW_OFF) < STACK_DEPTH * SW_FRAME)) return;
  WarpFrame& f = w_frame(sm, w.st);
  const int card = key_card(key), su = card_suit(card), r = card & 15, np8 = (int)(w.st & SW_NP8);
  const u32 bit = 1u << r, code = w.code, st = w.st, trick = w.trick, cards = w.all | w.now << 16;
  u32 info = (w.info & WI_KEEP) | key << 4;
  if (id.t < 16) f.m[id.t] = (uint16_t)w.m;
  if (id.s == su) {
    // The card's owner leaves the code: the owners of the cards below move up.
    const u32 low = 0xFFFFFFFFu >> (2 * w_popc(w.now >> r) - 2);
    w.code = (code & ~low) | (code << 2 & low);
    w.at |= bit << 16;
    w.now ^= bit;
  }
  if ((id.t & 15) == wi_seat(w.info) * 4 + su) w.m ^= bit;
  w.trick |= (u32)card << np8;
  if (np8 == 24) {
    const int c = (int)(w.trick >> (8 * (id.t & 3))) & 0xFF, cs = card_suit(c);
    const u32 rank = (cs == w.trump ? 512u : cs == card_suit((int)(w.trick & 0xFF)) ? 256u : 0u) | (u32)c << 2 | (u32)(id.t & 3);
    const u32 best = w_max(rank);
    const int wc = (int)(best >> 2) & 63, leader = (int)((st + best) & 3);
    const int same = w_popc(w_ballot(cs == card_suit(wc)) & 15);  // at least two: won by rank
    info |= (u32)(same >= 2 ? wc : 64) << 19;
    w.all = w.now;
    w.trick = 0;
    w.st = ((st & ~(SW_LEADER | SW_NP8)) | (u32)leader) + SW_FRAME - SW_LEFT - (ns_side(leader) ? SW_NEED : 0);
  } else {
    w.st = st + SW_CARD + SW_FRAME;
  }
  if (id.t < 4) {
    f.suit[id.t].at = w.at;
    f.suit[id.t].code = code;
    f.suit[id.t].cards = cards;
    f.suit[id.t].word = id.t == 0 ? st : id.t == 1 ? info : trick;
  }
  w_sync();
}

// Pops the top frame and takes its card back (node_done, unplay); returns the card.
DDG_W int w_unplay(WarpState& w, const WarpIds& id, WarpMem& sm) {
  const bool completed = (w.st & SW_NP8) == 0;  // this ply completed a trick
  if (!W_IN_BOUNDS((w.st & SW_OFF) - SW_FRAME < STACK_DEPTH * SW_FRAME)) return 0;
  const WarpFrame& f = w_frame(sm, w.st - SW_FRAME);
  w.st = f.suit[0].word;
  w.info = f.suit[1].word;
  w.trick = f.suit[2].word;
  w.at = f.suit[id.s].at;
  w.code = f.suit[id.s].code;
  const u32 cards = f.suit[id.s].cards;
  w.all = cards & 0xFFFFu;
  w.now = cards >> 16;
  w.m = f.m[id.t & 15];
  w_unpack(w);
  if (completed) {
    const int wc = wi_win_card(w.info);
    if (id.s == card_suit(wc)) w.rel |= 1u << (wc & 15);  // (none: suit 4)
  }
  return key_card(wi_key(w.info));
}

// The frame's next candidate (step_next): of those behind the last one, the first that is
// not a small card like one tried before; every candidate is tested by its thread. Returns
// its key, 0 when none is left.
DDG_W u32 w_next(WarpState& w, const WarpIds& id, WarpMem& sm) {
  if (!wi_more(w.info)) return 0;
  const u32 key = w_frame(sm, w.st).keys[id.t & 15];
  const int c = key_card(key);
  const u32 at = w_shfl(w.at, card_suit(c));
  const u32 acc = at & 0xFFFFu, tried = at >> 16, bit = 1u << (c & 15);
  const u32 small = (acc & (0u - acc)) - 1;  // below the lowest relevant card (all, when there is none)
  const bool skip = (small & bit) != 0 && (small & tried) != 0;
  return w_max(key < wi_key(w.info) && !skip ? key : 0);
}

// The top frame is done (finish): the relevant cards widen through runs of the hand's own
// touching cards.
DDG_W u32 w_widen(const WarpState& w, const WarpIds& id) {
  const u32 acc = w.at & 0xFFFFu, low = acc & (0u - acc);
  const u32 own = w_shfl(w.m, 4 * wi_seat(w.info) + id.s);
  const u32 below = w.all & (low - 1), stop = 2u << (w_top(below & ~own) & 31);  // (no stop: 2 << 31 = 0)
  return acc | (low & own ? below & (0u - (stop ? stop : 1u)) : 0);
}

// ---- root searches (start_search, start_lead, root_result) -----------------------------------

DDG_W void w_start_search(WarpState& w, const WarpJob& j, int target) {
  w.st = (u32)((j.decl + 1) & 3) | (u32)j.cards * SW_LEFT | (u32)target * SW_NEED;
  w.trick = 0;
}

// Starts the trick count of the current declarer: the binary search at `first`, or the
// stepping search from the seed `first`. (A deal has at least one card each, so every
// lead needs a search.)
DDG_W void w_start_lead(WarpState& w, const WarpIds& id, WarpJob& j, int first) {
  int lo = 0, hi = 13, target;
  if (j.mode == MODE_BISECT) {
    target = first < 1 ? 1 : first > 13 ? 13 : first;
  } else {
    lo = first < 0 ? 0 : first > j.cards ? j.cards : first;
    hi = lo == 0 ? PH_UP : PH_FIRST;
    target = lo == 0 ? 1 : lo;
  }
  w_start_search(w, j, target);
  w_sync();
  if (id.t == 0) {
    j.lo = (int8_t)lo;
    j.hi = (int8_t)hi;
  }
  w_sync();
}

// A root search at `target` finished with value v: the next target, or -1 with the answer
// in `lo`.
DDG_W int w_root_result(int mode, int cards, int target, int v, int& lo, int& hi) {
  if (mode == MODE_BISECT) {
    if (v) lo = target;
    else hi = target - 1;
    return lo < hi ? (lo + hi + 1) / 2 : -1;
  }
  if (hi == PH_DOWN || (hi == PH_FIRST && !v)) {  // going down: lo - 1 is next
    if (hi == PH_DOWN && v) return -1;
    hi = PH_DOWN;
    lo--;
    return lo > 0 ? lo : -1;
  }
  if (hi == PH_UP) {
    if (!v) return -1;
    lo++;
  }
  hi = PH_UP;
  return lo < cards ? lo + 1 : -1;
}

// Totals to shared memory: the node count and every thread's counter.
DDG_W void w_flush(WarpState& w, const WarpIds& id, WarpMem& sm) {
  if (id.t < WCNT_COUNT) sm.job.total[id.t] += w.cnt;
  if (id.t == 0) sm.job.nodes += w.nodes;
  w.cnt = 0;
  w.nodes = 0;
  w_sync();
}

// Ends the searcher after a failed bounds check.
DDG_W bool w_fault(WarpState& w, const WarpIds& id, WarpMem& sm) {
#ifdef DDG_BOUNDS_CHECK
  if (!w_any(w.fault)) return false;
  w_flush(w, id, sm);
  if (id.t == 0) sm.job.stage = ST_IDLE;
  w_sync();
  return true;
#else
  return false;
#endif
}

// A root search is done with value v and the root's cutting card `best` (or -1): the next
// search of the job, or its end (false).
template <class Env>
DDG_W bool w_end_root(WarpState& w, const WarpIds& id, WarpMem& sm, Env& env, int v, int best) {
  WarpJob& j = sm.job;
  if (best >= 0 && (v != 0) == ns_side(w.leader)) env.root_best(j, best);
  int lo = j.lo, hi = j.hi;
  const int next = w_root_result(j.mode, j.cards, w.need, v, lo, hi);
  w_sync();
  if (w_any(next >= 0)) {
    if (id.t == 0) {
      j.lo = (int8_t)lo;
      j.hi = (int8_t)hi;
    }
    w_sync();
    w_start_search(w, j, next);
    return true;
  }
  env.answer(j, lo);
  const int decl = j.decl + 1;
  w_sync();
  if (w_any(decl > j.last_decl)) {
    w_flush(w, id, sm);
    env.job_done(j);
    return false;
  }
  if (id.t == 0) j.decl = (int8_t)decl;
  w_sync();
  // The next lead starts at this answer (binary search) or at its own seed.
  w_start_lead(w, id, j, j.mode == MODE_BISECT ? lo : env.seed(j));
  return true;
}

// Runs jobs until none is left or the environment stops the warp. sm.job.stage: ST_TAKE to
// start with a job, ST_ENTER to go on inside one (w and the frames as they were saved); on
// return ST_IDLE (nothing left), ST_TAKE or ST_ENTER (stopped). An Env offers
//   bool take(w, id, sm)   the next job: position, job record (else stage is set)
//   bool stop(w, id, sm)   asked at a trick start after 256 nodes or more: true ends the warp
//   int seed(job), root_hint(job); void answer(job, ns), root_best(job, card), job_done(sm)
//   TTBucket* table(); u32 mask()
template <class Env>
DDG_W void w_run(WarpState& w, const WarpIds& id, WarpMem& sm, Env& env) {
  bool in_job = sm.job.stage == ST_ENTER, stopped = false;
  for (;;) {
    if (w_any(!in_job)) {
      if (!w_any(env.take(w, id, sm))) return;
      WarpJob& j = sm.job;
      w_start_lead(w, id, j, env.seed(j));
    }
    w.trump = (int)w_uni((u32)w.trump);
    // One node per turn: entered, then the frames it closes, up to the next card played.
    for (;;) {
      w.st = w_uni(w.st);
      w.trick = w_uni(w.trick);
      w_unpack(w);
      if (w.nplayed == 0 && W_RARE(w_any(w.nodes > 255u))) {
        w_flush(w, id, sm);
        if (env.stop(w, id, sm)) {
          stopped = true;
          break;
        }
      }
      w.nodes++;
      int hint = -1;
      bool store = false;
      WarpTop top = {0, 0};
      int v = w.nplayed == 0 ? w_lead(w, id, sm, env, store, top, hint) : w_enter_follow(w, id);
      if (w_fault(w, id, sm)) return;
      u32 key;  // the next card to play
      if (v < 0) {
        key = w_expand(w, id, sm, env, top, hint);
      } else {
        // The node is decided: its card is taken back, and the frames it completes with it.
        int best = -1;
        for (;;) {
          if (w_any(store)) w_put(w, id, sm, env, v, best);
          if (W_RARE((w.st & SW_OFF) == 0)) goto root_done;
          const int c = w_unplay(w, id, sm);
          if (w_fault(w, id, sm)) return;
          best = -1;
          if (w_any(v == (int)ns_side(wi_seat(w.info)))) {  // the child cuts
            w.at = (w.at & 0xFFFF0000u) | w.rel;
            best = c;
          } else {
            w.at |= w.rel;
            key = w_next(w, id, sm);
            if (key) break;
            v = wi_result(w.info);
          }
          w.rel = w_widen(w, id);
          store = w.nplayed == 0;
        }
        if (false) {
        root_done:
          in_job = w_end_root(w, id, sm, env, v, best);
          if (w_any(!in_job)) break;
          continue;
        }
      }
      if (w_fault(w, id, sm)) return;
      w_play(w, id, sm, key);
    }
    if (w_any(stopped)) return;
  }
}

}  // namespace ddg

#endif  // DDG_TT_SIG
