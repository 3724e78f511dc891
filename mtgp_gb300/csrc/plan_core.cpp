// plan_core.cpp -- see plan_core.h.  Flat arrays throughout: the per-item
// work is a few appends, so serving loops can plan thousands of requests
// per batch cheaply.
#include "plan_core.h"

#include <algorithm>
#include <cstdarg>
#include <cstdio>

namespace mtgp {

namespace {

int fail(std::string *err, int code, const char *fmt, ...) {
    char buf[200];
    va_list ap;
    va_start(ap, fmt);
    std::vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    if (err) *err = buf;
    return code;
}

// Piece lengths of cut runs are multiples of a grain: the largest power of
// two <= chunk / 8, at most 2^16 values.
uint64_t pieceGrain(uint64_t chunk) {
    uint64_t g = 1;
    while (g * 2 <= chunk / 8 && g < (uint64_t(1) << 16)) g *= 2;
    return g;
}

// The grain of plans whose chunk is the cheapest: 2^16, or 2^15 below chunks of
// 2^19.  The offsets are then multiples of it up to a run's length, few for a
// whole plan, and those of 2^16 are table polynomials: a plan's first launch
// makes no products for them.
uint64_t cheapGrain(uint64_t chunk) { return uint64_t(1) << (chunk >= uint64_t(1) << 19 ? 16 : 15); }

// A run: consecutive generated work of one stream starting at `start`.
struct Run {
    int32_t stream;
    uint64_t start, total;
    uint32_t first, n;  // segs of the run in the run-segment array
};

// How a run of `total` values is cut at chunk length `chunk`: k = ceil(total
// / chunk) near-equal pieces, rounded up to a multiple of the grain so that
// the pieces' offsets (and jump polynomials) recur across requests; the last
// piece takes the rest.  Returns the number of pieces (1: uncut).
uint64_t cutRun(uint64_t total, uint64_t chunk, uint64_t grain, uint64_t *piece) {
    *piece = total;
    if (chunk == 0 || total <= chunk) return 1;
    const uint64_t k = (total + chunk - 1) / chunk;
    *piece = ((total + k - 1) / k + grain - 1) / grain * grain;
    return (total + *piece - 1) / *piece;
}

// The chunk length with the shortest launch, for o.ctas CTAs per SM, in values
// generated by one of them (at MEXP 11213 0.59 ns a value on an SM with four,
// 0.42 with three, 0.30 with one or two, 32-bit; 1.0 ns with three or four and
// 0.75 with fewer, 64-bit):
//   - the jumps, one per piece but a run's first: o.jump_values each (85 and
//     107 ns on the whole GPU) after the o.jump_launch that the launch before
//     takes;
//   - the generation: the CTAs' even share of the values, or the long pieces
//     (over half of the longest) in the rounds that the CTAs need for them,
//     whichever is longer; the short ones fill what is left;
//   - with the grid of all resident CTAs (fewCtas): uncut runs that fit it at
//     once share an SM by that many, and of more tasks than few CTAs are for,
//     what is left of the longest one behind the even share runs nearly alone.
// Over 366 plans (1 to 10000 streams, lognormal, even and equal lengths, one
// kind and three, both word sizes, MEXP 11213 and 23209) the launch took 1.03
// of the time with the best of 12 lengths on average, 1.33 at most (1.04 and
// 1.37 without the last item, which 400 x 2^20 values at MEXP 23209 showed: 573
// us cut in two, 418 uncut).  Where no
// run is longer than jump_min nothing is cut: a pool without jumps needs no
// jump tables, which take longer to make than such a launch.
int64_t cheapestChunk(const std::vector<Run> &runs, uint64_t grand, const PlanOptions &o) {
    constexpr uint64_t kShortest = uint64_t(1) << 15;
    struct Cut {
        uint64_t k, piece, rest;
    };
    thread_local std::vector<uint64_t> longs;
    thread_local std::vector<Cut> cuts;
    longs.clear();
    uint64_t longest = 0;
    for (const Run &R : runs) {
        if (R.total > kShortest / 2) longs.push_back(R.total);
        longest = std::max(longest, R.total);
    }
    if (longest <= o.jump_min) return (int64_t)o.jump_min;
    const uint64_t slots = (uint64_t)o.ctas * (uint64_t)o.sms;
    const double share = (double)grand / (double)slots;
    // 4, 5, 6 and 7 times a power of two, from one above twice the even share
    // or one that cuts nothing down, until the jumps alone cost too much
    uint64_t base = kShortest / 4, m = 4;
    while (m * base < longest && (double)(m * base) <= 2 * share + (double)o.jump_min)
        if (++m == 8) base *= 2, m = 4;
    int64_t best = 0;
    double best_cost = 0;
    for (;;) {
        const uint64_t chunk = m * base, grain = cheapGrain(chunk);
        uint64_t jumps = 0, top = 0;
        cuts.clear();
        for (uint64_t t : longs) {
            uint64_t piece = t;
            if (t > chunk) {
                const uint64_t k = cutRun(t, chunk, grain, &piece);
                cuts.push_back({k, piece, t - (k - 1) * piece});
                jumps += k - 1;
            }
            top = std::max(top, piece);
        }
        const double jump_cost = (double)o.jump_values * (double)jumps +
                                 (jumps ? (double)o.jump_launch : 0);
        if (best && share + jump_cost > best_cost) return best;
        uint64_t nbig = 0;
        double big = 0;
        for (uint64_t t : longs)
            if (t <= chunk && 2 * t > top) nbig++, big += (double)t;
        for (const Cut &c : cuts) {
            if (2 * c.piece > top) nbig += c.k - 1, big += (double)((c.k - 1) * c.piece);
            if (2 * c.rest > top) nbig++, big += (double)c.rest;
        }
        const uint64_t tasks = runs.size() + jumps;
        const uint64_t per_sm = (tasks + (uint64_t)o.sms - 1) / (uint64_t)o.sms;
        const double slow = std::min(1.0, o.word_bytes == 4 ? std::max(0.5, (double)per_sm / o.ctas)
                                          : 2 * per_sm <= (uint64_t)o.ctas ? 0.75 : 1.0);
        const uint64_t rounds = (nbig + slots - 1) / slots;
        double gen = std::max(share, rounds <= 1 ? slow * (double)top
                                                 : (double)rounds * big / (double)nbig);
        if (tasks > kFewRounds * slots) {
            const double rate = (double)slots / (double)std::max<uint64_t>(o.resident, slots);
            gen = share + std::max(0.0, (double)top - rate * share) / 2;
        } else if (jumps == 0 && rounds > 1 && tasks <= (uint64_t)o.resident) {
            gen = std::max(share, (double)top * (double)per_sm / o.ctas);
        }
        if (!best || gen + jump_cost < best_cost) {
            best = (int64_t)chunk;
            best_cost = gen + jump_cost;
        }
        if (chunk == kShortest) return best;
        if (m-- == 4) base /= 2, m = 7;
    }
}

}  // namespace

int planCore(const mtgp_work_item_t *items, int nitems, const PlanOptions &o, PlanResult *r,
             std::string *err) {
    r->tasks.clear();
    r->segs.clear();
    r->stage_streams.clear();
    r->chunk = 0;
    r->out_bytes = 0;
    r->mode = -1;
    if (nitems < 0 || (nitems > 0 && !items))
        return fail(err, MTGP_ERR_INVALID, "bad item list (%d items)", nitems);
    // the items with work, grouped by stream in item order: keys (stream <<
    // 32 | item) sorted, so the cost follows the items, not the streams
    // (buffers are reused across calls of a thread: a server plans every
    // batch)
    thread_local std::vector<uint64_t> keys;
    keys.clear();
    for (int k = 0; k < nitems; k++) {
        const mtgp_work_item_t &it = items[k];
        if (it.stream >= (uint32_t)o.nstreams)
            return fail(err, MTGP_ERR_INVALID, "item %d: stream %u out of range", k,
                        (unsigned)it.stream);
        if (it.kind < -1 || it.kind > 4)
            return fail(err, MTGP_ERR_INVALID, "item %d: unknown kind %d", k, (int)it.kind);
        if (it.kind >= 0) {
            if (it.out_offset % o.word_bytes)
                return fail(err, MTGP_ERR_INVALID, "item %d: offset not a multiple of %llu", k,
                            (unsigned long long)o.word_bytes);
            if (it.count > (~uint64_t(0) - it.out_offset) / o.word_bytes)
                return fail(err, MTGP_ERR_INVALID, "item %d: output range overflows", k);
        }
        if (it.count == 0 && it.skip == 0) continue;
        keys.push_back((uint64_t)it.stream << 32 | (uint32_t)k);
    }
    if (keys.size() * 8 < (size_t)o.nstreams) {
        std::sort(keys.begin(), keys.end());
    } else {  // many items: a counting sort by stream (stable)
        thread_local std::vector<int32_t> head;
        thread_local std::vector<uint64_t> by;
        head.assign((size_t)o.nstreams + 1, 0);
        for (uint64_t key : keys) head[(key >> 32) + 1]++;
        for (int st = 0; st < o.nstreams; st++) head[st + 1] += head[st];
        by.resize(keys.size());
        for (uint64_t key : keys) by[(size_t)head[key >> 32]++] = key;
        keys.swap(by);
    }
    // runs, and the generated segments of each run
    thread_local std::vector<Run> runs;
    thread_local std::vector<PlanSeg> rseg;
    runs.clear();
    rseg.clear();
    rseg.reserve(keys.size() + 8);
    uint64_t grand = 0;
    for (size_t q0 = 0, q1; q0 < keys.size(); q0 = q1) {
        const int s = (int)(keys[q0] >> 32);
        for (q1 = q0; q1 < keys.size() && (int)(keys[q1] >> 32) == s; q1++) {
        }
        Run cur{s, 0, 0, (uint32_t)rseg.size(), 0};
        uint64_t pos = 0;
        for (size_t q = q0; q < q1; q++) {
            const int k = (int)(uint32_t)keys[q];
            const mtgp_work_item_t &it = items[k];
            uint64_t skip = it.skip, count = it.count;
            if (it.kind < 0) {  // advance only: all of it is a skip
                skip += count;
                count = 0;
                if (skip < it.skip) return fail(err, MTGP_ERR_INVALID, "item %d: skip overflows", k);
            }
            if (pos + skip < pos || pos + skip + count < pos + skip)
                return fail(err, MTGP_ERR_INVALID, "item %d: stream position overflows 64 bits", k);
            if (skip >= o.jump_min && o.can_jump) {
                if (cur.n) {
                    grand += cur.total;
                    runs.push_back(cur);
                }
                pos += skip;
                cur = Run{s, pos, 0, (uint32_t)rseg.size(), 0};
            } else if (skip) {
                if (skip > o.max_gen_skip)
                    return fail(err, MTGP_ERR_UNSUPPORTED,
                                "item %d: skip of %llu values would be generated (no in-kernel "
                                "jump for this exponent); jump the stream instead",
                                k, (unsigned long long)skip);
                rseg.push_back(PlanSeg{0, skip, -1, 0});
                cur.n++;
                cur.total += skip;
                pos += skip;
            }
            if (count) {
                const bool direct = o.direct && o.direct[k];
                rseg.push_back(PlanSeg{it.out_offset, count, it.kind, direct});
                cur.n++;
                cur.total += count;
                pos += count;
                if (!direct)
                    r->out_bytes = std::max(r->out_bytes, it.out_offset + count * o.word_bytes);
            }
        }
        if (cur.n || cur.start) {
            if (!cur.n) {  // ends with a jump: a task that only jumps
                rseg.push_back(PlanSeg{0, 0, -1, 0});
                cur.n = 1;
            }
            grand += cur.total;
            runs.push_back(cur);
        }
    }
    int64_t chunk = 0;
    if (o.can_jump) {
        if (o.chunk_tune > 0) {
            chunk = o.chunk_tune;
        } else if (o.chunk_tune == 0 && o.sms > 0) {
            chunk = cheapestChunk(runs, grand, o);
        } else if (o.chunk_tune == 0) {
            // a task longer than the average load of one CTA slot would set
            // the length of the whole launch
            const uint64_t per = grand / (uint64_t)std::max(o.resident, 1);
            chunk = (int64_t)std::max<uint64_t>(uint64_t(1) << 17, o.jump_min);
            while ((uint64_t)chunk < per) chunk <<= 1;
        }
    }
    // cut runs into tasks; per stream, mark write-back
    const bool cheap = o.sms > 0 && o.chunk_tune == 0;
    const uint64_t grain = chunk <= 0 ? 1
                           : cheap   ? cheapGrain((uint64_t)chunk)
                                     : pieceGrain((uint64_t)chunk);
    r->segs.reserve(rseg.size() + runs.size());
    bool cut = false;
    for (size_t r0 = 0, r1; r0 < runs.size(); r0 = r1) {
        for (r1 = r0; r1 < runs.size() && runs[r1].stream == runs[r0].stream; r1++) {
        }
        const size_t first_task = r->tasks.size();
        for (size_t ri = r0; ri < r1; ri++) {
            const Run &R = runs[ri];
            uint64_t piece;
            const uint64_t k = cutRun(R.total, chunk > 0 ? (uint64_t)chunk : 0, grain, &piece);
            if (k > 1) cut = true;
            uint32_t si = R.first;     // segment of R being cut
            const uint32_t se = R.first + R.n;
            uint64_t used = 0;         // values of it already taken
            for (uint64_t c = 0; c < k; c++) {
                PlanTask t{};
                t.stream = R.stream;
                t.run = R.start;
                t.off = c * piece;
                t.first = (uint32_t)r->segs.size();
                uint64_t want = (c + 1 == k) ? ~uint64_t(0) : piece;
                while (si < se && (want || rseg[si].count == used)) {
                    PlanSeg g = rseg[si];
                    const uint64_t take = std::min(g.count - used, want);
                    if (g.kind >= 0) g.out_off += used * o.word_bytes;
                    g.count = take;
                    r->segs.push_back(g);
                    t.total += take;
                    want -= take;
                    used += take;
                    if (used == rseg[si].count) {
                        si++;
                        used = 0;
                    }
                }
                t.n = (uint32_t)r->segs.size() - t.first;
                r->tasks.push_back(t);
            }
        }
        const size_t m = r->tasks.size() - first_task;
        for (size_t q = first_task; q < r->tasks.size(); q++)
            r->tasks[q].wb = m == 1 ? -1
                                    : (q + 1 == r->tasks.size() ? (int32_t)r->stage_streams.size()
                                                                : -2);
        if (m > 1) r->stage_streams.push_back(runs[r0].stream);
    }
    r->chunk = cut ? chunk : 0;
    // longest task first, a jump inside the kernel counted as jump_min
    // generated values (about its cost)
    const uint64_t jw = o.can_jump && o.sms == 0 ? o.jump_min : 0;
    auto cost = [jw](const PlanTask &t) {
        return t.total + jw * ((t.run ? 1u : 0u) + (t.off ? 1u : 0u));
    };
    // by (cost descending, position): a stable order, sorted as plain pairs
    thread_local std::vector<std::pair<uint64_t, uint32_t>> ord;
    thread_local std::vector<PlanTask> sorted;
    ord.resize(r->tasks.size());
    for (size_t q = 0; q < r->tasks.size(); q++)
        ord[q] = {~cost(r->tasks[q]), (uint32_t)q};
    std::sort(ord.begin(), ord.end());
    sorted.resize(r->tasks.size());
    for (size_t q = 0; q < ord.size(); q++) sorted[q] = r->tasks[ord[q].second];
    r->tasks.swap(sorted);
    int mode = -3;
    for (const PlanSeg &g : r->segs)
        if (g.count) mode = (mode == -3 || mode == g.kind) ? g.kind : -2;
    r->mode = mode == -3 ? -1 : mode;
    return MTGP_OK;
}

}  // namespace mtgp
