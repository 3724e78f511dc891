// plan_core.h -- host-side planning of one batched launch (no CUDA).
//
// Turns work items (mtgp_work_item_t: stream, kind, count, output offset,
// skip) into the tasks of a persistent launch.  Positions count steps from a
// stream's window at launch.
//   - Items of one stream keep the caller's order.
//   - A skip (or an advance-only item) of at least `jump_min` values, when
//     the kernels can jump (`can_jump`), is not generated: the work after it
//     is a new run that starts at that position, reached by jumping the
//     window inside the kernel.  Shorter skips are generated (advance items);
//     generated skips above `max_gen_skip` are rejected.
//   - A run longer than `chunk` is cut into k = ceil(length / chunk)
//     near-equal pieces whose length is rounded up to a multiple of the
//     largest power of two <= chunk / 8 (at most 2^16; the last piece takes
//     the rest); piece c starts at run start + c * piece.
//   - The chunk length is `chunk_tune` when > 0, none when < 0, and
//     otherwise the next power of two >= (all generated values / resident
//     CTAs), at least 2^17.
//   - The tasks of one stream all start from its window and run in
//     parallel.  A stream with one task writes its window back directly; with
//     several, the last one (in stream order) writes to a staging slot that is
//     copied back after the launch, the others write nothing.
//   - Tasks are ordered longest first, a start jump counting as `jump_min`
//     values (about its cost).
// The kernel-side jump of a task is X^run then X^off (either may be 0).
#pragma once
#include <cstddef>
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/mtgp_gpu.h"

namespace mtgp {

// First unit of part q of a jump split into `parts` over `tchunks` units
// (part q covers [partChunk(q), partChunk(q + 1))): every unit once, the
// earlier parts one more where they do not divide evenly.
inline int partChunk(int q, int tchunks, int parts) {
    const int rem = tchunks % parts;
    return q * (tchunks / parts) + (q < rem ? q : rem);
}

struct PlanOptions {
    int nstreams = 0;
    size_t word_bytes = 4;          // bytes of one output value
    bool can_jump = false;          // in-kernel jumps available
    uint64_t jump_min = uint64_t(1) << 17;
    uint64_t max_gen_skip = uint64_t(1) << 34;
    int64_t chunk_tune = 0;         // > 0 fixed, < 0 never cut, 0 automatic
    // per item: its out_offset is a device address, not an offset into the
    // output buffer (null: none is)
    const unsigned char *direct = nullptr;
    int resident = 1;               // resident CTAs of the jumping kernel
    // > 0: SMs of the GPU, for plans whose jumps are made ahead of the launch
    // and whose grid is `ctas` CTAs per SM; the automatic chunk is then the
    // cheapest (cheapestChunk), not a power of two.  jump_values: what a jump
    // costs, in values generated by one CTA; jump_launch: what the launch of
    // any number of them does
    int sms = 0, ctas = 4, jump_values = 150, jump_launch = 17000;
};

// CTAs per SM of a plan's launch where long runs set its length (fewCtas).
// Four of 11213's fill an SM's data pipe (4096
// lognormal streams of 32-bit words: 429 us on four, 456 on three and five,
// 625 on all ten that fit; 1024 streams of 64-bit words: 243 us, 264, 247,
// 356), and the fewer share it the sooner the longest tasks end.  Two of
// 23209's, which have twice the threads (512
// streams: 119 us on two, 144 on three, 168 on four).
inline int planCtas(int mexp) { return mexp == 11213 ? 4 : 2; }

// One item of a task: count values of kind (-1 = advance without output).
struct PlanSeg {
    uint64_t out_off;
    uint64_t count;
    int32_t kind;
    int32_t direct;
};

struct PlanTask {
    int32_t stream;
    int32_t wb;           // -1 = back to the stream, -2 = none, k >= 0 = staging slot k
    uint64_t run, off;    // start position = run + off
    uint64_t total;       // values the task steps through
    uint32_t first, n;    // its items: segs[first, first + n)
};

struct PlanResult {
    std::vector<PlanTask> tasks;        // longest first
    std::vector<PlanSeg> segs;
    std::vector<int32_t> stage_streams; // staging slot k -> stream
    int64_t chunk = 0;                  // chunk length used (0 = no run was cut)
    uint64_t out_bytes = 0;             // max over items of offset + size
    int mode = -1;                      // shared kind of all values, -1 all advance, -2 mixed
};

// Whether a plan runs on few CTAs per SM (planCtas) instead of all that fit.
// Few pay where the longest tasks set the launch's length: these are long, the
// tasks not so many that the work as a whole does, and the first of the second
// round is short beside the longest (equal tasks just over a round would take
// two).  Over 1150 plans of more tasks than few slots (to 10000 tasks; equal,
// lognormal and other lengths; every core but the four-word one; both
// exponents) few took 0.96 of the time of all (0.78 to 1.23) where this holds
// and 1.21 (0.87 to 2.3) where it does not:
//   4096 lognormal streams, median 65536     414 us on few, 428 on all
//   640 of 1 to 131071 values, 64-bit 23209   81            102
//   640 x 16384 (two rounds)                  24             19
//   10000 x 1000 (short tasks)                52             33
constexpr size_t kFewRounds = 8;
inline bool fewCtas(const PlanResult &r, const PlanOptions &o) {
    const size_t slots = (size_t)o.ctas * (size_t)o.sms, n = r.tasks.size();
    if (slots == 0 || n == 0 || n > kFewRounds * slots || r.tasks[0].total < o.jump_min / 2)
        return false;
    return n <= slots ||
           5 * (r.tasks[slots - 1].total + r.tasks[slots].total) <= 7 * r.tasks[0].total;
}

// Returns MTGP_OK or an MTGP_ERR_* code with a message in *err.
int planCore(const mtgp_work_item_t *items, int nitems, const PlanOptions &o, PlanResult *r,
             std::string *err);

}  // namespace mtgp
