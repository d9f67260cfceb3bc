// k_sweep.cu -- every overlap round of one or many read sets in ONE
// cooperative launch, many rounds per step.
//
// The entries of both tables stay where they are (no entry moves to another
// bin from round to round, as in k_bucket.cu); what a step of R rounds
// [r, r + R) finds is, for every entry, the round in which it is used.
//
//   A  every live suffix: its keys of the R rounds (NextSfx, overlap.cu:57-75)
//      into a Bloom filter (one 32-bit word, three bits per (round, key))
//   B  every live prefix: its R keys (PrevPfx, overlap.cu:77-91) against that
//      filter; a hit is a candidate: it enters a chain of its (key, round)'s
//      hash and a second, small filter
//   C  every live suffix again: its keys against the second filter, then the
//      chain; a suffix whose key is there makes a pair (suffix, prefix,
//      round) with each prefix of that key from another read (get_edges,
//      overlap.cu:557-603)
//   resolve  no entry was removed inside the step, so a pair may hold entries
//      that an earlier round of the step uses (remove_used, overlap.cu:694-710).
//      T[e] = the round that uses entry e is the one solution of
//        a pair matches iff T >= its round for both entries
//        T[e] = the smallest round of e's matching pairs, or never
//      found by iterating from T = never: after i iterations the first i
//      rounds are right, and statuses that no longer change are the solution.
//      An entry's nearest overlap is nearly always its partner's nearest too,
//      so a few iterations do, whatever R is.
//   commit  one record (key, entry, round) for each entry of a matching pair,
//      at most one per entry and job
//
// After the last step all records are grouped by (round, key range), each
// group sorted by (key, tie) -- the order of the reference's stable sort over
// its regenerated tables (overlap.cu:605-692) -- and joined; the edges go
// straight to their place in output.bin (overlap.cu:148-161).
//
// Why: the bucket kernel passes every live entry through a dozen block-wide
// phases in every round, which costs 15 us for a round of a few hundred
// entries and 42 us for one of a million.  Most live entries match in no
// round for a long time (an entry beyond a sequencing error or a coverage
// gap): here such an entry costs a hash step and three random L2 accesses
// per round, and a grid barrier is paid per phase of a step of up to 32
// rounds.  Bound: random accesses.  A lane's own line costs the load unit of
// an SM one cycle for a load (276 G/s on the chip), 1.5 for a reduction (188),
// 2.3 for an exchange (121), a sixth of that rate where they leave L2; a late
// step of 1.2M x 250 reads (16M keys) runs its reductions at 160 G/s and its
// loads at 160.  What is left around them: a chunk's entries (on their way a
// chunk ahead; its bases too gained nothing) and bases, the candidates' chain of an exchange and two
// stores, warps that end early (they draw their segments), and for a few
// thousand entries the latency of 8 barriers a step, 60 us.  All rounds,
// bucket kernel -> here: 2,000 x 100 reads 1.16 -> 0.245 ms, 100k x 150 1.90
// -> 0.505, 1.2M x 250 8.03 -> 3.17, 256 sets (13.2M reads) 71 -> 26 ms.
#include "coop_common.cuh"

namespace emp {

namespace {

constexpr int kST = kSweepThreads;      // 1024: one CTA per SM
constexpr int kSW = kST / 32;
constexpr uint32_t kNever = 0xffffffffu;
// (entry, round) keys of a step's first filters at most, and those up to which
// a key has 12 bits instead of 10.  Fewer keys a step would stay within L2 (a
// batch of 13.2M reads: 25M keys of 16 bits 29.8 ms, 56M of 12 26.2, 80M of 10
// 26.0, 112M of 12 27.4), but then every live entry is read and compacted for
// fewer rounds; fewer bits cost false candidates.
constexpr uint64_t kFilterKeys = 80u << 20, kFilterRoomy = 32u << 20;
constexpr uint32_t kU = 4;              // filter accesses of a lane in flight
constexpr uint32_t kQCap = 32 * (kU + 1);  // queued candidates per warp
constexpr uint32_t kBinMean = 32;       // matched entries per output bin aimed at
constexpr uint32_t kBinCap = 192;       // up to this many: one warp, in shared memory

struct SweepLoc {  // a job's step, the same in every CTA
    uint32_t r;          // first round of this step
    uint32_t R;          // rounds of this step
    uint32_t ls, lp;     // live suffixes and prefixes at its start
    uint32_t w1, w2;     // words of the two filters
    uint32_t cands;      // prefix candidates that the step found
    uint32_t pc, pairs;  // places up to the last one given to a candidate and a pair
    uint8_t act;         // the job runs this step
    uint8_t cur;         // key array that holds the keys of round r - 1
    uint8_t gm, gclean;  // log2 of the chain heads in use, and of those emptied so far
    uint8_t retry;       // the step before did not fit: its rounds again
};

struct SShared {
    uint32_t pref[kCoopMaxJobs + 1];
    uint32_t bin0[kCoopMaxJobs + 1];  // first output bin of each job
    SweepLoc loc[kCoopMaxJobs];
    uint32_t scan32[32];
    uint64_t scan64[32];
    uint64_t base;
    uint32_t flag, gen, pos, next;
    uint32_t fired[2 * kSweepMaxR];  // matched suffixes and prefixes by round of the step
    uint2 mult[4 * (kMaxReadLen + 1)];  // (enc * R^i) mod P of both fingerprints, enc = 1 .. 4
};

// A warp's part of the output phase: the records of one bin.
struct WarpBin {
    uint64_t sk[kBinCap];
    uint32_t val[kBinCap];
    uint32_t cnt[kBinCap];
    uint16_t ord[kBinCap];
};
constexpr size_t kQueueBytes = (size_t)kSW * kQCap * 16;
constexpr size_t kSweepWork = sizeof(WarpBin) * kSW > kQueueBytes ? sizeof(WarpBin) * kSW : kQueueBytes;
constexpr size_t kSweepShared = (sizeof(SShared) + 15) / 16 * 16;
constexpr size_t kSweepSmem = kSweepShared + kSweepWork;
// a chunk of an oversized bin's sort
constexpr uint32_t kBigChunk = kST;
static_assert(kBigChunk * 12 <= kSweepWork, "an oversized bin's chunk fits");

// ---------------------------------------------------------------- small pieces
// Reductions without a return value.  Through a pointer whose space the
// compiler does not know an atomicOr becomes an atomic that returns one (121
// against 188 G/s).
EMP_DEV void red_or(uint32_t *p, uint32_t v) {
    asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;\n" ::"l"(__cvta_generic_to_global(p)), "r"(v) : "memory");
}
EMP_DEV void red_min(uint32_t *p, uint32_t v) {
    asm volatile("red.relaxed.gpu.global.min.u32 [%0], %1;\n" ::"l"(__cvta_generic_to_global(p)), "r"(v) : "memory");
}
EMP_DEV uint32_t pow2_log(uint64_t n) {  // ceil(log2(n)), n >= 1
    return n <= 1 ? 0u : 64u - (uint32_t)__clzll(n - 1);
}
template <class S, class F>
EMP_DEV uint32_t sweep_prefix(S &sh, uint32_t *pref, int J, F count) {
    const uint32_t c = (int)threadIdx.x < J ? count((int)threadIdx.x) : 0u;
    uint32_t tot;
    const uint32_t ex = block_exclusive_scan<kST, uint32_t>(c, sh.scan32, &tot);
    if ((int)threadIdx.x < J) pref[threadIdx.x] = ex;
    if (threadIdx.x == 0) pref[J] = tot;
    __syncthreads();
    return tot;
}
EMP_DEV int job_of(const uint32_t *pref, int J, uint32_t t) {
    int lo = 0, hi = J;
    while (hi - lo > 1) {
        const int m = (lo + hi) >> 1;
        if (pref[m] <= t) lo = m;
        else hi = m;
    }
    return lo;
}

// (key, round of the step): 58 bits of fingerprints in order, 6 bits of round
EMP_DEV uint64_t pack_kq(uint32_t f1, uint32_t f2, uint32_t q) { return ((uint64_t)f1 << 35) | ((uint64_t)f2 << 6) | q; }
EMP_DEV uint32_t kq_f1(uint64_t k) { return (uint32_t)(k >> 35); }
EMP_DEV uint32_t kq_f2(uint64_t k) { return (uint32_t)(k >> 6) & kMask29; }
EMP_DEV uint32_t kq_q(uint64_t k) { return (uint32_t)k & 63u; }

// word and bits of (key, round) in a filter of `words` words
EMP_DEV uint32_t filter_mix(uint32_t f1, uint32_t f2, uint32_t q) {
    uint32_t h = f1 * 0x9E3779B1u + f2 * 0x85EBCA77u + q * 0xC2B2AE3Du;
    return h ^ (h >> 15);
}
EMP_DEV uint32_t filter_word(uint32_t h, uint32_t words) { return __umulhi(h * 0x2C1B3C6Du, words); }
EMP_DEV uint32_t filter_bits3(uint32_t h) {
    const uint32_t g = h * 0x297A2D39u;
    return (1u << (g >> 27)) | (1u << ((g >> 22) & 31u)) | (1u << ((g >> 17) & 31u));
}

// The bases that rounds r .. r + R - 1 drop from the entry's key, 2 bits
// each, first round lowest: a forward suffix or a reverse-complement prefix
// walks its read forwards from column r, the others backwards from L - 1 - r.
EMP_DEV uint64_t step_bases(const SweepJob &J, uint32_t val, uint32_t r, uint32_t R) {
    const uint32_t t = val >> 31, s = val & 1u;
    const bool inc = t == s;
    const uint32_t start = inc ? r : (uint32_t)J.L - r - R;
    const uint32_t *row = J.seq2 + (uint64_t)((val & 0x7fffffffu) >> 1) * J.wpr + (start >> 4);
    const uint32_t o = start & 15u, nw = (o + R + 15u) >> 4;  // 1 .. 3 words
    uint64_t x = __ldg(row);
    if (nw > 1) x |= (uint64_t)__ldg(row + 1) << 32;
    x >>= 2 * o;
    if (nw > 2) x |= (uint64_t)__ldg(row + 2) << (64 - 2 * o);  // o > 0 here
    if (!inc) {  // last column first
        uint64_t y = __brevll(x);
        y = ((y >> 1) & 0x5555555555555555ull) | ((y & 0x5555555555555555ull) << 1);
        x = y >> (64 - 2 * R);
    }
    return s ? x ^ 0xAAAAAAAAAAAAAAAAull : x;  // the complement's codes
}

// NextSfx on the two fingerprints: t = (enc * R^(len - 1)) mod P of both
EMP_DEV void step_sfx(uint32_t &f1, uint32_t &f2, uint2 t) {
    f1 = f1 >= t.x ? f1 - t.x : f1 + kP1 - t.x;
    f2 = f2 >= t.y ? f2 - t.y : f2 + kP2 - t.y;
}
EMP_DEV void step_pfx(uint32_t &f1, uint32_t &f2, uint32_t v, uint32_t inv1, uint32_t inv2) {
    const uint64_t k = prev_pfx(((uint64_t)f1 << 32) | f2, v, inv1, inv2);
    f1 = (uint32_t)(k >> 32);
    f2 = (uint32_t)k;
}

// ---------------------------------------------------------------- candidates
// chain of (key, round): the last candidate that entered it is the head
EMP_DEV uint32_t chain_hash(uint64_t k, uint32_t mask) { return (uint32_t)((k * 0x9E3779B97F4A7C15ull) >> 32) & mask; }

// Places of a step's candidates and pairs are handed out by 2^shard_log
// counters (all warps of the grid reach their flushes about together, and one
// counter takes 0.71 ns for each).  Runs of 32 places go round the counters,
// so that what a warp writes at once stays together.
EMP_DEV uint32_t shard_of(const SweepJob &J) { return blockIdx.x & ((1u << J.shard_log) - 1u); }
EMP_DEV uint32_t place(const SweepJob &J, uint32_t k, uint32_t p) {  // place p of counter k
    return (((p >> 5) << J.shard_log | k) << 5) | (p & 31u);
}
// whether place x has been given out; n: the counter that gives it
EMP_DEV const SweepShard &shard_at(const SweepJob &J, const SweepCtr &c, uint32_t x) {
    return c.shard[(x >> 5) & ((1u << J.shard_log) - 1u)];
}
EMP_DEV bool given(const SweepJob &J, uint32_t x, uint32_t n) { return (((x >> 5) >> J.shard_log) << 5 | (x & 31u)) < n; }

// T of iteration tg (numbered through the launch): word = (number
// complemented, 26 bits | round, 6 bits), so that atomicMin prefers the newer
// iteration and nothing is reset between iterations or steps.
constexpr uint32_t kClaimed = 62;  // round field of an entry whose record is written
EMP_DEV uint32_t t_word(uint32_t tg, uint32_t q) { return (~tg << 6) | q; }
EMP_DEV uint32_t t_round(uint32_t w, uint32_t tg) { return (w >> 6) == (~tg & 0x3ffffffu) ? w & 63u : kNever; }

// ---------------------------------------------------------------- a step's passes
struct Queue {  // a warp's candidates: (key, round), entry, value
    uint4 *q;
    uint32_t n;
};
EMP_DEV void queue_push(Queue &w, bool f, uint64_t kq, uint32_t e, uint32_t val) {
    const uint32_t m = __ballot_sync(0xffffffffu, f);
    if (!m) return;
    if (f) w.q[w.n + __popc(m & lanemask_lt_u32())] = make_uint4((uint32_t)kq, (uint32_t)(kq >> 32), e, val);
    w.n += __popc(m);
}

// up to 32 queued prefixes -> candidates, chains, second filter
EMP_DEV void flush_prefixes(SweepJob &J, SweepCtr &c, Queue &w, const SweepLoc &l) {
    const uint32_t lane = threadIdx.x & 31, n = w.n < 32u ? w.n : 32u;
    __syncwarp();
    const uint32_t at = w.n - n;
    uint32_t pos = 0;
    if (lane == 0) pos = atomicAdd(&c.shard[shard_of(J)].pc, n);
    pos = place(J, shard_of(J), __shfl_sync(0xffffffffu, pos, 0) + lane);
    if (lane < n) {
        const uint4 x = w.q[at + lane];
        if (pos < J.p_cap) {
            const uint64_t kq = (uint64_t)x.x | ((uint64_t)x.y << 32);
            const uint32_t next = atomicExch(J.heads + chain_hash(kq, (1u << l.gm) - 1u), pos);
            const uint32_t h = filter_mix(kq_f1(kq), kq_f2(kq), kq_q(kq));
            red_or(J.filter2 + filter_word(h, l.w2), filter_bits3(h));
            J.pcand[pos] = make_uint4(x.x, x.y, x.z, next);
        } else {
            c.ovf = 1;
        }
    }
    w.n = at;
    __syncwarp();
}

// up to 32 queued suffixes -> a pair with every prefix of another read with
// their key; the step's first T (nothing removed yet) from the pairs
EMP_DEV void flush_suffixes(SweepJob &J, SweepCtr &c, Queue &w, const SweepLoc &l, uint32_t tg) {
    const uint32_t lane = threadIdx.x & 31, n = w.n < 32u ? w.n : 32u;
    __syncwarp();
    const uint32_t at = w.n - n;
    uint4 x = make_uint4(0, 0, 0, 0);
    uint32_t p = kNever;
    if (lane < n) {
        x = w.q[at + lane];
        p = __ldcg(J.heads + chain_hash((uint64_t)x.x | ((uint64_t)x.y << 32), (1u << l.gm) - 1u));
    }
    uint32_t *const T = J.T[tg & 1u];
    const uint32_t walk = l.R > 1 ? 64u : 4096u, t = t_word(tg, x.x & 63u);
    for (uint32_t k = 0; __any_sync(0xffffffffu, p != kNever); ++k) {
        uint4 y = make_uint4(0, 0, 0, kNever);
        if (p != kNever) y = __ldcg(J.pcand + p);
        bool pair = p != kNever && y.x == x.x && y.y == x.y;
        uint32_t vp = 0;
        if (pair) {
            vp = __ldcg(J.val + y.z);
            pair = ((vp ^ x.w) & 0x7ffffffeu) != 0;
        }
        const uint32_t m = __ballot_sync(0xffffffffu, pair);
        if (m) {
            uint32_t pos = 0;
            if (lane == 0) pos = atomicAdd(&c.shard[shard_of(J)].pairs, (uint32_t)__popc(m));
            pos = place(J, shard_of(J), __shfl_sync(0xffffffffu, pos, 0) + __popc(m & lanemask_lt_u32()));
            if (pair && pos < J.pair_cap) {
                J.pair[pos] = make_uint4(x.x, x.y, x.w, vp);
                J.pair_e[pos] = make_uint2(x.z, y.z | 0x80000000u);
                red_min(T + x.z, t);
                red_min(T + y.z, t);
            }
            if (pair && pos >= J.pair_cap) c.ovf = 1;
        }
        p = y.w;
        if (k >= walk) {  // a crowded chain: fewer rounds at once, or another kernel
            c.ovf = 1;
            break;
        }
    }
    w.n = at;
    __syncwarp();
}

// One warp, one segment: drop the entries used in the step before (or before
// the launch) and move the rest to the segment's front in place.
// kPass 0: A, 1: B; pass 2 (C) finds the segment as A left it.  tg: number
// of the last iteration (the step before's T).
template <int kPass>
EMP_DEV void sweep_segment(SweepJob &J, const SweepLoc &l, SweepCtr &c, uint32_t seg, uint32_t b, uint32_t tg,
                           const uint2 *mult, Queue &w) {
    constexpr bool kPfx = kPass == 1;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t side0 = kPfx ? J.n_s : 0u, side_n = kPfx ? J.n_p : J.n_s;
    const uint32_t o = seg * J.seg, lim = side_n - o < J.seg ? side_n - o : J.seg;
    uint32_t *segcnt = J.segcnt + (kPfx ? J.segs_s : 0u) + seg;
    const uint32_t cnt = kPass != 2 && b == 0 ? lim : __ldcg(segcnt);
    const uint64_t e0 = (uint64_t)side0 + o;
    uint64_t *kin = J.key[l.cur], *kadv = J.key[l.cur ^ 1];
    // the first step's prefixes may be the suffixes' entries, read from there
    const bool half = kPfx && b == 0 && J.one_half;
    uint32_t *const T0 = J.T[0], *const T1 = J.T[1];
    const uint32_t *told = tg & 1u ? T1 : T0;
    uint32_t *const lval = J.val;
    const uint8_t *used = kPfx ? J.used_p : J.used_s;
    uint32_t *const filter = kPass == 2 ? J.filter2 : J.filter1;
    const uint32_t words = kPass == 2 ? l.w2 : l.w1, len0 = (uint32_t)J.L - l.r - 1u;
    const uint32_t inv1 = J.tables->inv1, inv2 = J.tables->inv2;
    const bool host_used = J.marked, stepped = J.stepped && l.r == (uint32_t)J.r0;  // in every try of the first step
    uint64_t *const win = J.bases + o;  // the suffixes' bases of the step, from pass A to pass C
    uint32_t live_n = 0;
    const uint64_t from = half ? e0 - side0 : e0;  // where the entries are read
    // the entries of the chunk after this one are on their way while it is worked on
    uint64_t nkey = 0, nbases = 0;
    uint32_t nval = 0, nold = kNever, nfull = 0;
    auto fetch = [&](uint32_t x) {
        if (kPass != 0) nfull = __ldcg(&c.ovf);
        if (x >= cnt) return;
        nkey = __ldcg(kin + from + x);
        nval = __ldcg(lval + from + x);
        if (kPass != 2 && b && !l.retry) nold = __ldcg(told + e0 + x);
        if (kPass == 2) nbases = __ldcg(win + x);
    };
    fetch(lane);
    for (uint32_t x0 = 0; x0 < cnt; x0 += 32) {
        const uint32_t x = x0 + lane;
        const uint64_t e = e0 + x;
        bool live = x < cnt;
        // the step does not fit and runs again: nothing more to find
        const uint32_t R = kPass != 0 && __any_sync(0xffffffffu, nfull) ? 0u : l.R;
        if (kPass == 2 && R == 0) break;
        const uint64_t key = nkey;
        const uint32_t val = nval | (half ? 0x80000000u : 0u);
        uint64_t bases = nbases;
        if (kPass != 2 && live) {
            if (b) live = t_round(nold, tg) == kNever;
            else if (host_used) live = used[val & 0x7fffffffu] == 0;
        }
        fetch(x + 32);
        uint64_t en = e;
        if (kPass != 2) {
            const uint32_t m = __ballot_sync(0xffffffffu, live);  // every lane has read its entry
            en = e0 + live_n + __popc(m & lanemask_lt_u32());
            live_n += __popc(m);
            __syncwarp();
            if (live && (en != e || half)) {
                lval[en] = val;
                kin[en] = key;
            }
            if (b == 0 && live) {  // no iteration's words yet
                T0[en] = kNever;
                T1[en] = kNever;
            }
        }
        uint32_t f1 = (uint32_t)(key >> 32), f2 = (uint32_t)key;
        if (kPass != 2 && live) {
            bases = step_bases(J, val, l.r, l.R);
            if (kPass == 0) win[en - e0] = bases;
        }
        for (uint32_t q0 = 0; q0 < R; q0 += kU) {
            uint32_t g1[kU], g2[kU], fw[kU];
#pragma unroll
            for (uint32_t u = 0; u < kU; ++u) {
                const uint32_t q = q0 + u;
                fw[u] = 0;
                if (q < R) {  // the same in every lane
                    const uint32_t v = (uint32_t)bases & 3u;
                    bases >>= 2;
                    if (u == 0 && q0 == 0 && stepped) {
                    } else if (kPfx) {
                        step_pfx(f1, f2, v, inv1, inv2);
                    } else {
                        step_sfx(f1, f2, mult[(len0 - q) * 4 + v]);
                    }
                    g1[u] = f1;
                    g2[u] = f2;
                    if (live) {
                        const uint32_t h = filter_mix(f1, f2, q);
                        if (kPass == 0) red_or(filter + filter_word(h, words), filter_bits3(h));
                        else fw[u] = __ldcg(filter + filter_word(h, words));
                    }
                }
            }
            if (kPass != 0) {
#pragma unroll
                for (uint32_t u = 0; u < kU; ++u) {
                    const uint32_t q = q0 + u;
                    if (q >= R) break;  // the same in every lane
                    const uint32_t bits = filter_bits3(filter_mix(g1[u], g2[u], q));
                    const bool hit = live && (fw[u] & bits) == bits;
                    queue_push(w, hit, pack_kq(g1[u], g2[u], q), (uint32_t)en, val);
                }
                while (w.n >= 32) {
                    if (kPass == 1) flush_prefixes(J, c, w, l);
                    else flush_suffixes(J, c, w, l, tg + 1);
                }
            }
        }
        if (kPass != 0 && live) kadv[en] = ((uint64_t)f1 << 32) | f2;
    }
    if (kPass != 2 && lane == 0) {
        *segcnt = live_n;
        if (b == 0 && host_used) atomicAdd(kPfx ? &c.lp : &c.ls, live_n);
    }
}

// Pass kPass of the step over every live segment of the active jobs, one warp
// per segment.
template <int kPass>
EMP_DEV void sweep_pass(SweepJob *jobs, int J, uint32_t b, uint32_t tg, SShared &sh, uint8_t *smem) {
    if (threadIdx.x == 0) sh.next = 0;
    const uint32_t total = sweep_prefix(sh, sh.pref, J, [&](int j) -> uint32_t {
        if (!sh.loc[j].act) return 0u;
        return kPass == 1 ? jobs[j].segs_p : jobs[j].segs_s;
    });
    const uint32_t warp = threadIdx.x >> 5;
    Queue w{reinterpret_cast<uint4 *>(smem) + warp * kQCap, 0u};
    int j = -1;
    auto drain = [&]() {
        if (kPass == 0 || j < 0) return;
        while (kPass != 0 && w.n) {
            if (kPass == 1) flush_prefixes(jobs[j], jobs[j].ctr[b % 3], w, sh.loc[j]);
            else flush_suffixes(jobs[j], jobs[j].ctr[b % 3], w, sh.loc[j], tg + 1);
        }
    };
    // neighbouring segments to different SMs, an SM's to its warps as they come free
    for (;;) {
        uint32_t t = 0;
        if ((threadIdx.x & 31) == 0) t = atomicAdd(&sh.next, 1u);
        t = __shfl_sync(0xffffffffu, t, 0) * gridDim.x + blockIdx.x;
        if (t >= total) break;
        const int jn = job_of(sh.pref, J, t);
        if (jn != j) drain();
        j = jn;
        sweep_segment<kPass>(jobs[j], sh.loc[j], jobs[j].ctr[b % 3], t - sh.pref[j], b, tg, sh.mult, w);
    }
    drain();
}

// ---------------------------------------------------------------- resolving a step
// A pair (suffix, prefix, round q) matches iff both entries are live in round
// q: T >= q.  Its status (bit 31 of the prefix's entry: it matches) starts
// as true; iteration tg takes it from T[tg - 1] and T[tg] is the smallest
// round of each entry's matching pairs.  When no status changes T[tg] = T[tg
// - 1] is the solution.
EMP_DEV void resolve_pairs(SweepJob *jobs, int J, uint32_t b, uint32_t tg, uint32_t *chg, SShared &sh) {
    const uint32_t total = sweep_prefix(sh, sh.pref, J, [&](int j) -> uint32_t {
        return sh.loc[j].act ? (sh.loc[j].pairs + kST - 1) / kST : 0u;
    });
    bool changed = false;
    for (uint32_t t = blockIdx.x; t < total; t += gridDim.x) {
        const int j = job_of(sh.pref, J, t);
        SweepJob &jb = jobs[j];
        const uint32_t x = (t - sh.pref[j]) * kST + threadIdx.x;
        if (x >= sh.loc[j].pairs) continue;
        const uint32_t given_n = __ldcg(&shard_at(jb, jb.ctr[b % 3], x).pairs);
        const uint32_t q = __ldcg(reinterpret_cast<const uint32_t *>(jb.pair + x)) & 63u;
        const uint2 e = __ldcg(jb.pair_e + x);
        if (!given(jb, x, given_n)) continue;
        const uint32_t ep = e.y & 0x7fffffffu;
        const uint32_t *T0 = jb.T[(tg - 1) & 1u];
        uint32_t *T1 = jb.T[tg & 1u];
        const uint32_t ts = __ldcg(T0 + e.x), tp = __ldcg(T0 + ep);
        const bool on = t_round(ts, tg - 1) >= q && t_round(tp, tg - 1) >= q;
        if (on) {
            red_min(T1 + e.x, t_word(tg, q));
            red_min(T1 + ep, t_word(tg, q));
        }
        if (on != (e.y >> 31 != 0)) {
            changed = true;
            jb.pair_e[x].y = on ? ep | 0x80000000u : ep;
        }
    }
    if (__syncthreads_or(changed) && threadIdx.x == 0) atomicOr(chg, 1u);
}

// Append one record for every thread with f set to those at *ctr: the
// thread's position.  Called by the whole CTA.
EMP_DEV uint32_t block_append(uint32_t f, uint32_t *ctr, SShared &sh) {
    uint32_t tot;
    const uint32_t ex = block_exclusive_scan<kST, uint32_t>(f, sh.scan32, &tot);
    if (threadIdx.x == 0) sh.pos = tot ? atomicAdd(ctr, tot) : 0u;
    __syncthreads();
    const uint32_t p = sh.pos + ex;
    __syncthreads();
    return p;
}

// The step's matching pairs: a record for each of their entries (the first
// pair of an entry claims it), the counts per round; chains emptied, filters
// zeroed.
EMP_DEV void commit_step(SweepJob *jobs, int J, uint32_t b, uint32_t tg, SShared &sh) {
    uint32_t total = sweep_prefix(sh, sh.pref, J, [&](int j) -> uint32_t {
        return sh.loc[j].act ? (sh.loc[j].pairs + kST - 1) / kST : 0u;
    });
    for (uint32_t t = blockIdx.x; t < total; t += gridDim.x) {
        const int j = job_of(sh.pref, J, t);
        SweepJob &jb = jobs[j];
        SweepCtr &c = jb.ctr[b % 3];
        for (uint32_t k = threadIdx.x; k < 2 * kSweepMaxR; k += kST) sh.fired[k] = 0;
        __syncthreads();
        const uint32_t x = (t - sh.pref[j]) * kST + threadIdx.x;
        uint4 v = make_uint4(0, 0, 0, 0);
        bool fs = false, fp = false;
        if (x < sh.loc[j].pairs) {
            const uint32_t given_n = __ldcg(&shard_at(jb, c, x).pairs);
            const uint2 e = __ldcg(jb.pair_e + x);
            if (given(jb, x, given_n) && e.y >> 31) {
                v = __ldcg(jb.pair + x);
                uint32_t *T = jb.T[tg & 1u];
                fs = (atomicExch(T + e.x, t_word(tg, kClaimed)) & 63u) != kClaimed;
                fp = (atomicExch(T + (e.y & 0x7fffffffu), t_word(tg, kClaimed)) & 63u) != kClaimed;
            }
        }
        const uint64_t kq = (uint64_t)v.x | ((uint64_t)v.y << 32);
        const uint32_t q = kq_q(kq), r = sh.loc[j].r;
        if (fs) atomicAdd(&sh.fired[q], 1u);
        if (fp) atomicAdd(&sh.fired[kSweepMaxR + q], 1u);
        uint32_t p = block_append((uint32_t)fs + (uint32_t)fp, &jb.nrec, sh);
        if (fs) jb.rec[p++] = make_uint4(kq_f2(kq), kq_f1(kq), v.z, r + q);
        if (fp) jb.rec[p] = make_uint4(kq_f2(kq), kq_f1(kq), v.w, r + q);
        if (threadIdx.x < 2 * kSweepMaxR) {  // two warps: the suffixes' counts, the prefixes'
            const uint32_t f = sh.fired[threadIdx.x];
            if (f) atomicAdd((threadIdx.x < kSweepMaxR ? jb.fs : jb.fp) + r + (threadIdx.x & (kSweepMaxR - 1)), f);
            const uint32_t all = __reduce_add_sync(0xffffffffu, f);
            if ((threadIdx.x & 31) == 0 && all) atomicAdd(threadIdx.x < kSweepMaxR ? &c.fired_s : &c.fired_p, all);
        }
        __syncthreads();
    }
    total = sweep_prefix(sh, sh.pref, J, [&](int j) -> uint32_t {
        if (!sh.loc[j].act) return 0u;
        return (sh.loc[j].pc + kST - 1) / kST;
    });
    for (uint32_t t = blockIdx.x; t < total; t += gridDim.x) {  // every chain has a candidate
        const int j = job_of(sh.pref, J, t);
        SweepJob &jb = jobs[j];
        const uint32_t x = (t - sh.pref[j]) * kST + threadIdx.x;
        if (x < sh.loc[j].pc) {
            const uint32_t given_n = __ldcg(&shard_at(jb, jb.ctr[b % 3], x).pc);
            const uint2 k = __ldcg(reinterpret_cast<const uint2 *>(jb.pcand + x));
            if (!given(jb, x, given_n)) continue;
            jb.heads[chain_hash((uint64_t)k.x | ((uint64_t)k.y << 32), (1u << sh.loc[j].gm) - 1u)] = kNever;
        }
    }
}

// chain heads that no step of the job has used yet: emptied
EMP_DEV void clean_heads(SweepJob *jobs, int J, SShared &sh) {
    constexpr uint32_t kTile = kST * 16;  // heads per tile: four 16-byte stores a thread
    const uint32_t total = sweep_prefix(sh, sh.pref, J, [&](int j) -> uint32_t {
        const SweepLoc &l = sh.loc[j];
        if (!l.act || l.gm <= l.gclean) return 0u;
        const uint32_t lo = l.gclean ? 1u << l.gclean : 0u;
        return ((1u << l.gm) - lo + kTile - 1) / kTile;
    });
    for (uint32_t t = blockIdx.x; t < total; t += gridDim.x) {
        const int j = job_of(sh.pref, J, t);
        const SweepLoc &l = sh.loc[j];
        const uint32_t lo = (l.gclean ? 1u << l.gclean : 0u) + (t - sh.pref[j]) * kTile, hi = min(lo + kTile, 1u << l.gm);
        for (uint32_t i = lo + 4 * threadIdx.x; i < hi; i += 4 * kST)  // all multiples of four
            *reinterpret_cast<uint4 *>(jobs[j].heads + i) = make_uint4(kNever, kNever, kNever, kNever);
    }
}

// zero the words that the step used of both filters
EMP_DEV void clear_filters(SweepJob *jobs, int J, SShared &sh) {
    constexpr uint32_t kWords = kST * 16;  // per tile: four 16-byte stores a thread
    const uint32_t total = sweep_prefix(sh, sh.pref, J, [&](int j) -> uint32_t {
        const SweepLoc &l = sh.loc[j];
        return l.act ? (l.w1 + kWords - 1) / kWords + (l.w2 + kWords - 1) / kWords : 0u;
    });
    for (uint32_t t = blockIdx.x; t < total; t += gridDim.x) {
        const int j = job_of(sh.pref, J, t);
        const SweepLoc &l = sh.loc[j];
        uint32_t k = t - sh.pref[j];
        const uint32_t t1 = (l.w1 + kWords - 1) / kWords;
        uint32_t *f = k < t1 ? jobs[j].filter1 : jobs[j].filter2;
        const uint32_t words = k < t1 ? l.w1 : l.w2;
        if (k >= t1) k -= t1;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t i = k * kWords + (u * kST + threadIdx.x) * 4;
            if (i < words) *reinterpret_cast<uint4 *>(f + i) = make_uint4(0, 0, 0, 0);
        }
    }
}

// ---------------------------------------------------------------- output
// ex[i] = sum of in[0 .. i) for i <= n (global arrays; in[n] unused), over the
// whole grid: chunk sums, a barrier, then every CTA scans its chunk.
template <class In>
EMP_DEV bool grid_scan(const In *in, uint64_t *ex, uint32_t n, uint64_t *part, CoopCtl *ctl, SShared &sh) {
    const uint32_t per = (n + gridDim.x - 1) / gridDim.x;
    const uint32_t lo = min(n, blockIdx.x * per), hi = min(n, lo + per);
    uint64_t sum = 0;
    for (uint32_t i = lo + threadIdx.x; i < hi; i += kST) sum += __ldcg(in + i);
    uint64_t tot;
    block_exclusive_scan<kST, uint64_t>(sum, sh.scan64, &tot);
    if (threadIdx.x == 0) part[blockIdx.x] = tot;
    if (!grid_barrier_raw(ctl, &sh.flag, &sh.gen)) return false;
    uint64_t before = 0;
    for (uint32_t i = threadIdx.x; i < blockIdx.x; i += kST) before += __ldcg(part + i);
    uint64_t run;
    block_exclusive_scan<kST, uint64_t>(before, sh.scan64, &run);
    for (uint32_t i0 = lo; i0 < hi; i0 += kST) {
        const uint32_t i = i0 + threadIdx.x;
        const uint64_t v = i < hi ? (uint64_t)__ldcg(in + i) : 0;
        const uint64_t x = block_exclusive_scan<kST, uint64_t>(v, sh.scan64, &tot);
        if (i < hi) ex[i] = run + x;
        run += tot;
    }
    if (hi == n && lo < hi && threadIdx.x == 0) ex[n] = run;
    if (n == 0 && blockIdx.x == 0 && threadIdx.x == 0) ex[0] = 0;
    return grid_barrier_raw(ctl, &sh.flag, &sh.gen);
}

EMP_DEV uint32_t tie_key(uint32_t val) {  // rid parity, then read (the regenerated tables' order)
    const uint32_t rid = val & 0x7fffffffu;
    return ((rid & 1u) << 31) | (rid >> 1);
}
EMP_DEV bool rec_before(uint64_t ska, uint32_t va, uint64_t skb, uint32_t vb) {
    return ska < skb || (ska == skb && tie_key(va) < tie_key(vb));
}
EMP_DEV uint64_t rec_sk(const uint4 &x) { return sort_key((uint64_t)x.x | ((uint64_t)x.y << 32), x.z); }
// output bin of a record within its job: the round's bins in key order
EMP_DEV uint32_t rec_bin(const SweepJob &J, const uint4 &x) {
    const uint32_t k = x.w - (uint32_t)J.r0;
    const uint32_t b0 = __ldcg(J.binbase + k), nb = __ldcg(J.binbase + k + 1) - b0;
    return b0 + bkt_of(rec_sk(x), nb);
}

// A job's rounds from the counts of matched entries: table sizes, the rounds
// that run (overlap.cu:258), output bins.  One CTA; rounds <= kST.
EMP_DEV void round_sizes(SweepJob &J, SShared &sh) {
    const uint32_t nr = (uint32_t)(J.rounds - J.r0), t = threadIdx.x;
    const uint32_t fs = t < nr ? __ldcg(J.fs + J.r0 + t) : 0u, fp = t < nr ? __ldcg(J.fp + J.r0 + t) : 0u;
    uint32_t ts, tp, tb, tr;
    const uint32_t es = block_exclusive_scan<kST, uint32_t>(fs, sh.scan32, &ts);
    const uint32_t ep = block_exclusive_scan<kST, uint32_t>(fp, sh.scan32, &tp);
    const uint32_t s0 = J.marked ? vld(J.s0) : J.n_s, p0 = J.marked ? vld(J.p0) : J.n_p;
    const uint32_t S = s0 - es, P = p0 - ep;
    block_exclusive_scan<kST, uint32_t>(t < nr && S > 0 ? 1u : 0u, sh.scan32, &tr);
    const uint32_t c = fs + fp;
    const uint32_t bx = block_exclusive_scan<kST, uint32_t>((c + kBinMean - 1) / kBinMean, sh.scan32, &tb);
    if (t < nr) {
        J.binbase[t] = bx;
        RoundRecord &x = J.records[J.r0 + t];
        x.S = S;
        x.P = P;
        x.C = c;
        x.nb = (c + kBinMean - 1) / kBinMean;
    }
    if (t == 0) {
        J.binbase[nr] = tb;
        J.nbins = tb;
        J.round = (uint32_t)J.r0 + tr;
    }
    __syncthreads();
}

// A job's edges per round and the records' places in its output.  One CTA.
EMP_DEV void round_places(SweepJob &J, uint32_t bin0, const uint64_t *eoff, SShared &sh) {
    const uint32_t nr = vld(J.round) - (uint32_t)J.r0, t = threadIdx.x;
    uint64_t E = 0, e0 = 0, bytes = 0, P = 0;
    if (t < nr) {
        e0 = __ldcg(eoff + bin0 + __ldcg(J.binbase + t));
        E = __ldcg(eoff + bin0 + __ldcg(J.binbase + t + 1)) - e0;
        P = __ldcg(&J.records[J.r0 + t].P);
        bytes = P ? 12 + 8 * E : 0;
    }
    const uint64_t all = __ldcg(eoff + bin0 + vld(J.nbins)) - __ldcg(eoff + bin0);
    uint64_t tot;
    const uint64_t off = block_exclusive_scan<kST, uint64_t>(bytes, sh.scan64, &tot);
    if (t == 0) {
        J.e_total = all;
        if (all > J.ecap) J.overflow = 1;
    }
    if (t < nr) {
        RoundRecord &x = J.records[J.r0 + t];
        x.E = E;
        x.e0 = e0 - __ldcg(eoff + bin0);
        J.roff[t] = off;
        if (P && all <= J.ecap) {  // u64 n, i32 ovlp_len (write_edges_binary, overlap.cu:148-161)
            uint32_t *h = reinterpret_cast<uint32_t *>(J.out + off);
            h[0] = (uint32_t)E;
            h[1] = (uint32_t)(E >> 32);
            h[2] = (uint32_t)(J.L - 1 - J.r0 - (int)t);
        }
    }
    __syncthreads();
}

// One bin by one warp: its records sorted by (sort key, tie) into `sorted`
// with each suffix's edge count; returns the bin's edges.
EMP_DEV uint32_t sort_bin_warp(const uint4 *in, uint4 *sorted, uint32_t c, WarpBin &w) {
    const uint32_t lane = threadIdx.x & 31;
    __syncwarp();
    for (uint32_t i = lane; i < c; i += 32) {
        const uint4 x = __ldcg(in + i);
        w.sk[i] = rec_sk(x);
        w.val[i] = x.z;
    }
    __syncwarp();
    for (uint32_t i = lane; i < c; i += 32) {
        const uint64_t sk = w.sk[i];
        const uint32_t v = w.val[i];
        uint32_t rk = 0;
        for (uint32_t k = 0; k < c; ++k) rk += rec_before(w.sk[k], w.val[k], sk, v);
        w.ord[rk] = (uint16_t)i;
    }
    __syncwarp();
    uint32_t edges = 0;
    for (uint32_t i = lane; i < c; i += 32) {
        const uint32_t a = w.ord[i], va = w.val[a];
        const uint64_t ka = w.sk[a];
        uint32_t cc = 0;
        if (!(va >> 31))
            for (uint32_t k = i + 1; k < c; ++k) {
                const uint32_t o = w.ord[k], vo = w.val[o];
                if ((w.sk[o] >> 1) != (ka >> 1)) break;
                cc += (vo >> 31) && ((vo & 0x7fffffffu) >> 1) != ((va & 0x7fffffffu) >> 1);
            }
        edges += cc;
        // the key back from the sort key: fp1 = bits 30.., fp2 = bits 1..29
        sorted[i] = make_uint4((uint32_t)(ka >> 1) & kMask29, (uint32_t)(ka >> 30), va, cc);
    }
    return __reduce_add_sync(0xffffffffu, edges);
}

// the sorted bin's edges at from[o ..], to[o ..] by one warp
EMP_DEV void write_bin_warp(const uint4 *sorted, uint32_t c, uint32_t *from, uint32_t *to, uint64_t o, WarpBin &w) {
    const uint32_t lane = threadIdx.x & 31;
    __syncwarp();
    for (uint32_t i = lane; i < c; i += 32) {
        const uint4 x = __ldcg(sorted + i);
        w.sk[i] = (uint64_t)x.x | ((uint64_t)x.y << 32);
        w.val[i] = x.z;
        w.cnt[i] = x.w;
    }
    __syncwarp();
    for (uint32_t i0 = 0; i0 < c; i0 += 32) {
        const uint32_t i = i0 + lane;
        const uint32_t n = i < c ? w.cnt[i] : 0u;
        uint32_t x = n;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
            if ((int)lane >= d) x += y;
        }
        if (n) {
            uint64_t at = o + x - n;
            const uint32_t va = w.val[i];
            uint32_t left = n;
            for (uint32_t k = i + 1; left; ++k) {
                const uint32_t vo = w.val[k];
                if ((vo >> 31) && ((vo & 0x7fffffffu) >> 1) != ((va & 0x7fffffffu) >> 1)) {
                    from[at] = va & 0x7fffffffu;
                    to[at] = vo & 0x7fffffffu;
                    ++at;
                    --left;
                }
            }
        }
        o += __shfl_sync(0xffffffffu, x, 31);
    }
}

// The same for a bin of more than kBinCap records by a whole CTA: chunks of
// kBigChunk ranked by comparing all pairs, then every record adds, per other
// chunk, the records before it (binary search).  `in` is left chunk-sorted.
EMP_DEV uint64_t sort_bin_cta(uint4 *in, uint4 *sorted, uint32_t c, SShared &sh, uint8_t *smem) {
    uint64_t *sk = reinterpret_cast<uint64_t *>(smem);
    uint32_t *vv = reinterpret_cast<uint32_t *>(sk + kBigChunk);
    for (uint32_t lo = 0; lo < c; lo += kBigChunk) {
        const uint32_t m = min(c - lo, kBigChunk);
        uint4 x = make_uint4(0, 0, 0, 0);
        if (threadIdx.x < m) {
            x = __ldcg(in + lo + threadIdx.x);
            sk[threadIdx.x] = rec_sk(x);
            vv[threadIdx.x] = x.z;
        }
        __syncthreads();
        if (threadIdx.x < m) {
            const uint64_t k = sk[threadIdx.x];
            uint32_t rk = 0;
            for (uint32_t u = 0; u < m; ++u) rk += rec_before(sk[u], vv[u], k, x.z);
            in[lo + rk] = x;
        }
        __syncthreads();
    }
    for (uint32_t i = threadIdx.x; i < c; i += kST) {
        const uint4 x = __ldcg(in + i);
        const uint64_t k = rec_sk(x);
        uint32_t rk = i % kBigChunk;
        for (uint32_t lo = 0; lo < c; lo += kBigChunk) {
            if (lo == i / kBigChunk * kBigChunk) continue;
            uint32_t a = 0, z = min(c - lo, kBigChunk);
            while (a < z) {
                const uint32_t mid = (a + z) >> 1;
                const uint4 y = __ldcg(in + lo + mid);
                if (rec_before(rec_sk(y), y.z, k, x.z)) a = mid + 1;
                else z = mid;
            }
            rk += a;
        }
        sorted[rk] = make_uint4(x.x, x.y, x.z, 0u);
    }
    __syncthreads();
    uint64_t edges = 0;
    for (uint32_t i = threadIdx.x; i < c; i += kST) {
        const uint4 x = __ldcg(sorted + i);
        if (x.z >> 31) continue;
        uint32_t cc = 0;
        for (uint32_t k = i + 1; k < c; ++k) {
            const uint4 y = __ldcg(sorted + k);
            if (y.x != x.x || y.y != x.y) break;
            cc += (y.z >> 31) && ((y.z & 0x7fffffffu) >> 1) != ((x.z & 0x7fffffffu) >> 1);
        }
        edges += cc;
        reinterpret_cast<uint32_t *>(sorted + i)[3] = cc;
    }
    uint64_t tot;
    block_exclusive_scan<kST, uint64_t>(edges, sh.scan64, &tot);
    return tot;
}
EMP_DEV void write_bin_cta(const uint4 *sorted, uint32_t c, uint32_t *from, uint32_t *to, uint64_t o, SShared &sh) {
    for (uint32_t i0 = 0; i0 < c; i0 += kST) {
        const uint32_t i = i0 + threadIdx.x;
        uint4 x = make_uint4(0, 0, 0, 0);
        if (i < c) x = __ldcg(sorted + i);
        uint64_t tot;
        uint64_t at = o + block_exclusive_scan<kST, uint64_t>((uint64_t)x.w, sh.scan64, &tot);
        uint32_t left = x.w;
        for (uint32_t k = i + 1; left; ++k) {
            const uint32_t vo = __ldcg(reinterpret_cast<const uint32_t *>(sorted + k) + 2);
            if ((vo >> 31) && ((vo & 0x7fffffffu) >> 1) != ((x.z & 0x7fffffffu) >> 1)) {
                from[at] = x.z & 0x7fffffffu;
                to[at] = vo & 0x7fffffffu;
                ++at;
                --left;
            }
        }
        o += tot;
    }
}

// What pass B and C of a job's step found, in one read of its counters.
EMP_DEV void step_counts(const SweepJob &J, const SweepCtr &c, SweepLoc &l) {
    const uint32_t last = (1u << J.shard_log) - 1u, ovf = __ldcg(&c.ovf);
    uint2 n = __ldcg(reinterpret_cast<const uint2 *>(&c.shard[0]));
    uint32_t all = n.x, mc = n.x, mp = n.y;
    if (last) {
        uint2 v[kSweepShards];
#pragma unroll
        for (uint32_t k = 1; k < kSweepShards; ++k)  // in flight together
            v[k] = __ldcg(reinterpret_cast<const uint2 *>(&c.shard[min(k, last)]));
#pragma unroll
        for (uint32_t k = 1; k < kSweepShards; ++k) {
            all += k <= last ? v[k].x : 0u;
            mc = max(mc, v[k].x);
            mp = max(mp, v[k].y);
        }
    }
    l.cands = all;
    l.pc = min(((mc + 31) & ~31u) << J.shard_log, J.p_cap);
    l.pairs = ovf ? 0u : min(((mp + 31) & ~31u) << J.shard_log, J.pair_cap);
}

// the job's step after step b - 1: its first round, its length, its chains
EMP_DEV void next_step(SweepJob &J, SweepLoc &l, uint32_t b) {
    if (!l.act) return;
    const SweepCtr &c = J.ctr[(b - 1) % 3];
    l.gclean = max(l.gclean, l.gm);
    if (b == 1 && J.marked) {  // counted by the first step
        l.ls = __ldcg(&c.ls);
        l.lp = __ldcg(&c.lp);
    }
    l.retry = __ldcg(&c.ovf) != 0;
    if (l.retry) {  // too many candidates: the same rounds again, fewer at once
        if (l.R == 1) {
            l.act = 0;
            if (blockIdx.x == 0) J.crowded = 1;
        }
        l.R = l.R > 4 ? l.R / 4 : 1u;
        return;
    }
    const uint32_t us = __ldcg(&c.fired_s), up = __ldcg(&c.fired_p);
    // about one candidate per live entry and step, were none removed
    const uint64_t want = us ? (uint64_t)l.ls * l.R / us : (uint64_t)kSweepMaxR;
    const uint64_t tried = (uint64_t)l.lp * l.R, cands = l.cands;
    l.ls -= us;
    l.lp -= up;
    l.r += l.R;
    l.cur ^= 1;
    uint32_t R = (uint32_t)(want < 4ull * l.R ? want : 4ull * l.R);
    R = R < 1 ? 1u : R > (uint32_t)kSweepMaxR ? (uint32_t)kSweepMaxR : R;
    const uint32_t left = (uint32_t)J.rounds > l.r ? (uint32_t)J.rounds - l.r : 0u;
    l.R = R < left ? R : left;
    l.act = left > 0 && l.ls > 0 && l.lp > 0;
    // a chain per candidate that the last step's rate gives
    const uint32_t gm = pow2_log(cands * ((uint64_t)l.lp * l.R) / (tried ? tried : 1) + 1024);
    l.gm = (uint8_t)min(gm, (uint32_t)J.gm_max);
}
// filter sizes of a step, its rounds cut so that all jobs' first filters stay
// within kFilterKeys keys (all = live suffixes of all jobs)
EMP_DEV void size_filters(const SweepJob &J, SweepLoc &l, uint64_t all) {
    const uint64_t cap = all ? kFilterKeys / all : 1;
    if (l.R > cap) l.R = cap < 1 ? 1u : (uint32_t)cap;
    while (l.R > 1 && (uint64_t)l.ls * l.R > 4ull * J.w1_max) l.R = (l.R + 1) / 2;  // 8 bits per key where memory ends
    const uint64_t keys = (uint64_t)l.ls * l.R;
    const uint64_t w = all * l.R <= kFilterRoomy ? (keys * 3 + 7) / 8 : (keys * 5 + 15) / 16;
    l.w1 = (uint32_t)(w < 1024 ? 1024 : w < J.w1_max ? (w + 3) / 4 * 4 : J.w1_max);
    l.w2 = l.w1 > 4096 ? (l.w1 / 4 + 3) / 4 * 4 : 1024;
}

// Profiling aid: at the end of a phase, (phase | step << 8, job 0's first
// round and rounds of the step, its candidates) and the time.
struct SweepTrace {
    CoopCtl *ctl;
    uint32_t n;
};
EMP_DEV void mark(SweepTrace &t, uint32_t phase, uint32_t b, const SShared &sh) {
    if (!t.ctl->trace || blockIdx.x != 0 || threadIdx.x != 0 || t.n >= t.ctl->trace_cap) return;
    uint64_t *p = t.ctl->trace + (uint64_t)t.n * kCoopTracePhases;
    p[0] = phase | (uint64_t)b << 8;
    p[1] = sh.loc[0].r | (uint64_t)sh.loc[0].R << 32;
    p[2] = sh.loc[0].cands | (uint64_t)sh.loc[0].pairs << 32;
    p[3] = globaltimer();
    p[4] = sh.loc[0].ls | (uint64_t)sh.loc[0].lp << 32;
    ++t.n;
}

__global__ void __launch_bounds__(kST, 1) sweep_kernel(SweepJob *jobs, CoopCtl *ctl, SweepOut go, int zero) {
    extern __shared__ __align__(16) uint8_t smem_all[];
    SShared &sh = *reinterpret_cast<SShared *>(smem_all);
    uint8_t *smem = smem_all + kSweepShared;
    const int J = (int)ctl->njobs;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (uint32_t i = tid; i < 4 * (kMaxReadLen + 1); i += kST) {
        const uint64_t e = (i & 3) + 1;
        sh.mult[i] = make_uint2(mod1(e * jobs[0].tables->pow1[i >> 2]), mod2(e * jobs[0].tables->pow2[i >> 2]));
    }
    if (tid == 0) sh.gen = 0;
    if (tid < J) {
        const SweepJob &x = jobs[tid];
        SweepLoc &l = sh.loc[tid];
        l.r = (uint32_t)x.r0;
        l.ls = x.n_s;
        l.lp = x.n_p;
        const uint32_t left = x.rounds > x.r0 ? (uint32_t)(x.rounds - x.r0) : 0u;
        l.R = min(left, x.first_r);
        l.act = left > 0 && x.n_s > 0;
        l.retry = 0;
        l.cur = x.cur0;
        l.gclean = 0;
        l.gm = (uint8_t)min(pow2_log((uint64_t)x.n_p / 2 + 1024), (uint32_t)x.gm_max);
    }
    __syncthreads();
    SweepTrace tr{ctl, 0u};
    mark(tr, 0, 0, sh);
    if (zero) {
        const uint32_t total = sweep_prefix(sh, sh.pref, J, [&](int j) -> uint32_t { return (jobs[j].zeroed + 4 * kST - 1) / (4 * kST); });
        for (uint32_t t = blockIdx.x; t < total; t += gridDim.x) {
            const int j = job_of(sh.pref, J, t);
            uint4 *p = reinterpret_cast<uint4 *>(jobs[j].filter1);
            const uint32_t lo = (t - sh.pref[j]) * 4 * kST, hi = min(lo + 4 * kST, jobs[j].zeroed);
            for (uint32_t i = lo + tid; i < hi; i += kST) p[i] = make_uint4(0, 0, 0, 0);
        }
        if (!grid_barrier_raw(ctl, &sh.flag, &sh.gen)) return;
    }
    uint32_t tg = 0;  // resolving iterations of the launch
    for (uint32_t b = 0;; ++b) {
        if (b && tid < J) next_step(jobs[tid], sh.loc[tid], b);
        uint64_t all;
        block_exclusive_scan<kST, uint64_t>(tid < J && sh.loc[tid].act ? (uint64_t)sh.loc[tid].ls : 0ull, sh.scan64, &all);
        if (tid < J) size_filters(jobs[tid], sh.loc[tid], all);
        if (!__syncthreads_or(tid < J && sh.loc[tid].act)) break;
        mark(tr, 1, b, sh);
        uint32_t *chg = go.chg + (b % 3) * kSweepIters;
        clean_heads(jobs, J, sh);
        sweep_pass<0>(jobs, J, b, tg, sh, smem);
        if (!grid_barrier_raw(ctl, &sh.flag, &sh.gen)) return;
        mark(tr, 2, b, sh);
        sweep_pass<1>(jobs, J, b, tg, sh, smem);
        if (!grid_barrier_raw(ctl, &sh.flag, &sh.gen)) return;
        mark(tr, 3, b, sh);
        if (blockIdx.x == gridDim.x - 1) {  // the next step's counters (last read two steps ago)
            for (uint32_t k = tid; k < (uint32_t)J * kSweepShards; k += kST) {
                SweepShard &x = jobs[k / kSweepShards].ctr[(b + 1) % 3].shard[k % kSweepShards];
                x.pc = x.pairs = 0;
            }
            if (tid < J) {
                SweepCtr &c = jobs[tid].ctr[(b + 1) % 3];
                c.ls = c.lp = c.ovf = c.fired_s = c.fired_p = 0;
                if (b == 0 && jobs[tid].marked) {
                    jobs[tid].s0 = __ldcg(&jobs[tid].ctr[0].ls);
                    jobs[tid].p0 = __ldcg(&jobs[tid].ctr[0].lp);
                }
            }
            if (tid < kSweepIters) go.chg[((b + 1) % 3) * kSweepIters + tid] = 0;
        }
        sweep_pass<2>(jobs, J, b, tg, sh, smem);
        if (!grid_barrier_raw(ctl, &sh.flag, &sh.gen)) return;
        mark(tr, 4, b, sh);
        ++tg;  // the T of the pairs as pass C found them: final where every step is one round
        if (tid < J && sh.loc[tid].act) step_counts(jobs[tid], jobs[tid].ctr[b % 3], sh.loc[tid]);
        if (__syncthreads_or(tid < J && sh.loc[tid].act && sh.loc[tid].R > 1 && sh.loc[tid].pairs)) {
            for (uint32_t it = 0; it < (uint32_t)kSweepIters; ++it) {  // kSweepMaxR + 1 suffice
                resolve_pairs(jobs, J, b, ++tg, chg + it, sh);
                if (!grid_barrier_raw(ctl, &sh.flag, &sh.gen)) return;
                mark(tr, 5, b, sh);
                if (!__ldcg(chg + it)) break;
            }
        }
        clear_filters(jobs, J, sh);
        commit_step(jobs, J, b, tg, sh);
        if (!grid_barrier_raw(ctl, &sh.flag, &sh.gen)) return;
        mark(tr, 6, b, sh);
    }
    // ---- output: the rounds' sizes, the records by (round, key range)
    for (int j = blockIdx.x; j < J; j += gridDim.x) round_sizes(jobs[j], sh);
    if (!grid_barrier_raw(ctl, &sh.flag, &sh.gen)) return;
    mark(tr, 11, 0, sh);
    const uint32_t nb = sweep_prefix(sh, sh.bin0, J, [&](int j) -> uint32_t { return vld(jobs[j].nbins); });
    uint32_t tiles = sweep_prefix(sh, sh.pref, J, [&](int j) -> uint32_t { return (vld(jobs[j].nrec) + kST - 1) / kST; });
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int j = job_of(sh.pref, J, t);
        const uint32_t x = (t - sh.pref[j]) * kST + tid;
        if (x < vld(jobs[j].nrec))
            jobs[j].rank[x] = atomicAdd(go.cnt + sh.bin0[j] + rec_bin(jobs[j], __ldcg(jobs[j].rec + x)), 1u);
    }
    if (!grid_barrier_raw(ctl, &sh.flag, &sh.gen)) return;
    mark(tr, 12, 0, sh);
    if (!grid_scan(go.cnt, go.off, nb, go.part, ctl, sh)) return;
    mark(tr, 20, 0, sh);
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int j = job_of(sh.pref, J, t);
        const uint32_t x = (t - sh.pref[j]) * kST + tid;
        if (x < vld(jobs[j].nrec)) {
            const uint4 v = __ldcg(jobs[j].rec + x);
            const uint64_t at = __ldcg(go.off + sh.bin0[j] + rec_bin(jobs[j], v)) - __ldcg(go.off + sh.bin0[j]);
            jobs[j].rec2[at + __ldcg(jobs[j].rank + x)] = v;
        }
    }
    if (!grid_barrier_raw(ctl, &sh.flag, &sh.gen)) return;
    mark(tr, 13, 0, sh);
    WarpBin &wb = reinterpret_cast<WarpBin *>(smem)[warp];
    for (uint32_t t = warp * gridDim.x + blockIdx.x; t < nb; t += gridDim.x * kSW) {
        const int j = job_of(sh.bin0, J, t);
        const uint32_t c = __ldcg(go.cnt + t);
        const uint64_t at = __ldcg(go.off + t) - __ldcg(go.off + sh.bin0[j]);
        uint32_t e = 0;
        if (c) {
            if (lane == 0) go.round[t] = __ldcg(&jobs[j].rec2[at].w);
            if (c <= kBinCap) e = sort_bin_warp(jobs[j].rec2 + at, jobs[j].rec + at, c, wb);
            else if (lane == 0) go.big[atomicAdd(go.nbig, 1u)] = t;
        }
        if (lane == 0 && c <= kBinCap) go.ecnt[t] = e;
    }
    if (!grid_barrier_raw(ctl, &sh.flag, &sh.gen)) return;
    mark(tr, 14, 0, sh);
    const uint32_t nbig = vld(*go.nbig);
    if (nbig) {
        for (uint32_t k = blockIdx.x; k < nbig; k += gridDim.x) {
            const uint32_t t = __ldcg(go.big + k);
            const int j = job_of(sh.bin0, J, t);
            const uint64_t at = __ldcg(go.off + t) - __ldcg(go.off + sh.bin0[j]);
            const uint64_t e = sort_bin_cta(jobs[j].rec2 + at, jobs[j].rec + at, __ldcg(go.cnt + t), sh, smem);
            if (tid == 0) go.ecnt[t] = e;
            __syncthreads();
        }
        if (!grid_barrier_raw(ctl, &sh.flag, &sh.gen)) return;
    mark(tr, 15, 0, sh);
    }
    if (!grid_scan(go.ecnt, go.eoff, nb, go.part, ctl, sh)) return;
    mark(tr, 21, 0, sh);
    for (int j = blockIdx.x; j < J; j += gridDim.x) round_places(jobs[j], sh.bin0[j], go.eoff, sh);
    if (!grid_barrier_raw(ctl, &sh.flag, &sh.gen)) return;
    mark(tr, 16, 0, sh);
    auto place_bin = [&](uint32_t t, int &j, uint32_t *&from, uint32_t *&to, uint64_t &o, uint64_t &at) -> bool {
        j = job_of(sh.bin0, J, t);
        const SweepJob &jb = jobs[j];
        if (vld(jb.overflow)) return false;
        const uint32_t k = __ldcg(go.round + t) - (uint32_t)jb.r0;
        const uint64_t E = __ldcg(&jb.records[jb.r0 + k].E);
        o = __ldcg(go.eoff + t) - __ldcg(go.eoff + sh.bin0[j] + __ldcg(jb.binbase + k));
        from = reinterpret_cast<uint32_t *>(jb.out + __ldcg(jb.roff + k) + 12);
        to = from + E;
        at = __ldcg(go.off + t) - __ldcg(go.off + sh.bin0[j]);
        return true;
    };
    for (uint32_t t = warp * gridDim.x + blockIdx.x; t < nb; t += gridDim.x * kSW) {
        const uint32_t c = __ldcg(go.cnt + t);
        if (!c || c > kBinCap) continue;
        int j;
        uint32_t *from, *to;
        uint64_t o, at;
        if (place_bin(t, j, from, to, o, at)) write_bin_warp(jobs[j].rec + at, c, from, to, o, wb);
    }
    __syncthreads();
    for (uint32_t k = blockIdx.x; k < nbig; k += gridDim.x) {
        const uint32_t t = __ldcg(go.big + k);
        int j;
        uint32_t *from, *to;
        uint64_t o, at;
        if (place_bin(t, j, from, to, o, at)) write_bin_cta(jobs[j].rec + at, __ldcg(go.cnt + t), from, to, o, sh);
    }
}

size_t al(size_t x) { return (x + 255) / 256 * 256; }

}  // namespace

uint32_t sweep_segment_size(uint64_t entries_per_side) {
    // one segment per warp of the grid up to 1024 entries, then several of 512
    // or fewer that the warps draw (batch of 256, 5 segments of 1024 a warp in
    // fixed turns 33.2 ms, drawn 30.5; of 512 29.8; of 256 30.8)
    const uint64_t per = (entries_per_side + 148ull * kSW - 1) / (148ull * kSW);
    const uint64_t waves = per <= 1024 ? 1 : (per + 512 - 1) / 512;
    const uint64_t s = ((per + waves - 1) / waves + 31) / 32 * 32;
    return (uint32_t)(s < 32 ? 32 : s);
}

// a job of `entries` of a launch's entries per side: its share of the warps
// that draw places, and none for a few thousand entries
uint32_t sweep_shard_log(uint64_t entries, uint64_t entries_per_side) {
    uint32_t k = 0;
    while ((2u << k) <= kSweepShards && (2ull << k) * entries_per_side <= kSweepShards * entries &&
           (8192ull << k) <= entries)
        ++k;
    return k;
}

// Rounds of a job's first step, for about one candidate per entry: U unique
// keys among n2 read-ends give the reads that start at a base and strand
// (lambda; U / n2 = (1 - e^-lambda) / lambda of them differ), and an entry
// finds a partner in a round with nearly that probability.  A dense set's
// step that does not fit runs again with fewer rounds.
uint32_t sweep_first_rounds(uint64_t U, uint64_t n2) {
    const double d = n2 > U ? 1.0 - (double)U / (double)n2 : 0.0;
    const double lambda = 2.0 * d * (1.0 + d * (2.0 / 3.0));
    const double r = lambda > 0 ? 0.8 / lambda : 4.0;
    return r < 1.0 ? 1u : r > 4.0 ? 4u : (uint32_t)r;
}

uint32_t sweep_bins_max(uint64_t n_in, int rounds) { return (uint32_t)(n_in / kBinMean) + (uint32_t)rounds + 1; }

// One job's work memory from `base` (null: only the size); its first *zeroed
// bytes are to be zero at the launch.
size_t sweep_layout(uint8_t *base, SweepJob *J, size_t *zeroed) {
    size_t o = 0;
    auto take = [&](size_t bytes) -> uint8_t * {
        uint8_t *p = base ? base + o : nullptr;
        o = al(o + bytes);
        return p;
    };
    const uint64_t ns = J->n_s, np = J->n_p, n = ns + np;
    const int rounds = J->rounds;
    // filter 1 holds twelve rounds of every suffix at 10 bits each
    const uint64_t w1 = ns < 256 ? 1024 : 4 * ns < (1u << 24) ? 4 * ns : 1u << 24;
    J->w1_max = (uint32_t)w1;
    uint32_t gm = 10;
    while ((1ull << gm) < np) ++gm;
    J->gm_max = gm;
    // a quarter more than every shard's share
    J->p_cap = (uint32_t)(((np + np / 4) >> J->shard_log) / 32 + 2) << (J->shard_log + 5);
    J->pair_cap = (uint32_t)(((n + n / 4) >> J->shard_log) / 32 + 2) << (J->shard_log + 5);
    J->segs_s = (uint32_t)((ns + J->seg - 1) / J->seg);
    J->segs_p = (uint32_t)((np + J->seg - 1) / J->seg);
    J->filter1 = reinterpret_cast<uint32_t *>(take((size_t)4 * w1));
    J->filter2 = reinterpret_cast<uint32_t *>(take((size_t)4 * (w1 > 4096 ? w1 / 4 + 4 : 1024)));
    J->ctr = reinterpret_cast<SweepCtr *>(take(3 * sizeof(SweepCtr)));
    J->fs = reinterpret_cast<uint32_t *>(take((size_t)rounds * 4));
    J->fp = reinterpret_cast<uint32_t *>(take((size_t)rounds * 4));
    *zeroed = o;
    J->zeroed = (uint32_t)(o / 16);
    J->heads = reinterpret_cast<uint32_t *>(take((size_t)4 << gm));
    J->bases = reinterpret_cast<uint64_t *>(take(ns * 8));
    for (int k = 0; k < 2; ++k) J->T[k] = reinterpret_cast<uint32_t *>(take(n * 4));
    J->segcnt = reinterpret_cast<uint32_t *>(take((size_t)(J->segs_s + J->segs_p) * 4));
    J->pcand = reinterpret_cast<uint4 *>(take((size_t)J->p_cap * 16));
    J->pair = reinterpret_cast<uint4 *>(take((size_t)J->pair_cap * 16));
    J->pair_e = reinterpret_cast<uint2 *>(take((size_t)J->pair_cap * 8));
    J->rec = reinterpret_cast<uint4 *>(take(n * 16));
    J->rec2 = reinterpret_cast<uint4 *>(take(n * 16));
    J->rank = reinterpret_cast<uint32_t *>(take(n * 4));
    J->binbase = reinterpret_cast<uint32_t *>(take((size_t)(rounds + 1) * 4));
    J->roff = reinterpret_cast<uint64_t *>(take((size_t)(rounds + 1) * 8));
    return o;
}

size_t sweep_out_layout(uint8_t *base, uint32_t bins, SweepOut *go, size_t *zeroed) {
    size_t o = 0;
    auto take = [&](size_t bytes) -> uint8_t * {
        uint8_t *p = base ? base + o : nullptr;
        o = al(o + bytes);
        return p;
    };
    SweepOut g;
    g.chg = reinterpret_cast<uint32_t *>(take(3 * kSweepIters * 4));
    g.nbig = reinterpret_cast<uint32_t *>(take(4));
    g.cnt = reinterpret_cast<uint32_t *>(take((size_t)bins * 4));
    *zeroed = o;
    g.off = reinterpret_cast<uint64_t *>(take((size_t)(bins + 1) * 8));
    g.ecnt = reinterpret_cast<uint64_t *>(take((size_t)bins * 8));
    g.eoff = reinterpret_cast<uint64_t *>(take((size_t)(bins + 1) * 8));
    g.round = reinterpret_cast<uint32_t *>(take((size_t)bins * 4));
    g.big = reinterpret_cast<uint32_t *>(take((size_t)bins * 4));
    g.part = reinterpret_cast<uint64_t *>(take(1024 * 8));
    *go = g;
    return o;
}

static int sweep_grid_find(int dev) {
    int sms = 0, coop = 0, occ = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop) return 0;
    if (cudaFuncSetAttribute(sweep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSweepSmem) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, sweep_kernel, kST, kSweepSmem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return occ >= 1 && sms <= 1024 ? sms : 0;  // one CTA per SM
}

int sweep_grid_size() {
    constexpr int kDevs = 64;
    static std::atomic<int> grid[kDevs] = {};  // grid + 1; 0: not found yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevs) {
        cudaGetLastError();
        return sweep_grid_find(dev);
    }
    int g = grid[dev].load(std::memory_order_relaxed);
    if (g == 0) {
        g = sweep_grid_find(dev) + 1;
        grid[dev].store(g, std::memory_order_relaxed);
    }
    return g - 1;
}

cudaError_t launch_sweep(SweepJob *jobs, CoopCtl *ctl, const SweepOut &go, bool zero, cudaStream_t s) {
    const int grid = sweep_grid_size();
    if (grid <= 0) return cudaErrorNotSupported;
    SweepOut g = go;
    int z = zero ? 1 : 0;
    void *args[] = {&jobs, &ctl, &g, &z};
    count_launch();
    return cudaLaunchCooperativeKernel((const void *)sweep_kernel, dim3(grid), dim3(kST), args, kSweepSmem, s);
}

}  // namespace emp
