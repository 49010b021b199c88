// stroke_verbs.h — launch interface of the verb-parallel stroke (stroke_verbs.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "kernels.h"

namespace lg {

// Device arrays of the verb-parallel stroke, one entry per verb of the batch ("slot": the verb's
// index less the batch's first) unless said otherwise. Filled by the count phase, read by the
// emit phase.
struct StrokeVerbs {
    uint32_t cap;          // verbs the arrays have room for (vpre and ipre: one entry more)
    float4* firsts;        // the verb's first two kept points
    float4* adv;           // advancements (stroke_steps.cu): at the verb's last four kept points, .w
                           // the last; for records of a verb of two runs .x at the join between
    float4* lasts;         // the kept point before the verb's last one, and the one before that
    float2* fin;           // its last kept point, where that is not its end point
    uint32_t* rec;         // first point of the verb; End/Close: the slot of the sub-path's Begin
    uint32_t* path;
    uint32_t* join;        // the general join at the verb's end point (packed counts and ids)
    uint32_t* split;       // the join between the two runs of a verb that has two
    uint32_t* drops;       // list of verbs whose end point merged (before `split` is written)
    uint32_t* cut;         // where that join is
    uint32_t* extra;       // list of the verbs that have one
    uint32_t* irregular;   // list of the irregular verbs
    uint32_t* vpre;        // vertices of the batch before this verb (its own until the scan)
    uint32_t* ipre;        // indices, likewise
    uint16_t* flags;
    uint8_t* kind;
    uint32_t* path_walk;   // per path: not 0 when the path is left to the walk of stroke.cu
    uint32_t* walk_list;   // those paths
    uint32_t* path_v;      // per path: vpre and ipre of its first verb
    uint32_t* path_i;
    uint32_t* words;       // [0] verbs of the batch, [1] offsets out of order, [2] paths in
                           // walk_list, [3] some verb has interior steps, [4] drops, [5] scan tile,
                           // [6] extra, [7] irregular, [STROKE_VERBS_UNFIT] as [1], for the kernels
    unsigned long long* scan;  // tile states, after the words
    size_t clear_bytes;    // words and tile states, cleared by every count phase
};
constexpr uint32_t STROKE_VERBS_READ = 4;    // words the host reads back
constexpr uint32_t STROKE_VERBS_WORDS = 64;  // words in all
// A word that every warp reads, on a 128-byte line without the counters: beside them walk_kernel
// took 66 instead of 50 us for 1,000 paths of 16 segments.
constexpr uint32_t STROKE_VERBS_UNFIT = 32;
// Bytes per verb of the arrays above, for their allocation.
constexpr size_t STROKE_VERBS_BYTES = 3 * 16 + 8 + 9 * 4 + 2 + 1;

// Streams for kernels that run beside those of the caller's stream: fork(i, s) returns a stream
// that continues after what is on `s`, join(i, s) makes `s` wait for it. Without streams (none
// could be made) the work goes on `s` itself.
struct SideStreams {
    static constexpr int N = 3;
    cudaStream_t stream[N] = {};
    cudaEvent_t forked[N] = {}, joined[N] = {};
    cudaStream_t fork(int i, cudaStream_t s) const {
        if (!stream[i]) return s;
        cudaEventRecord(forked[i], s);
        cudaStreamWaitEvent(stream[i], forked[i], 0);
        return stream[i];
    }
    void join(int i, cudaStream_t s) const {
        if (!stream[i]) return;
        cudaEventRecord(joined[i], stream[i]);
        cudaStreamWaitEvent(s, joined[i], 0);
    }
};

// What follows the counts of a batch of few paths, in the same launch: the index range per path, the
// paths' places, and the totals.
constexpr uint32_t STROKE_FINISH_PATHS = 2048;
struct StrokeFinish {
    uint64_t *vtx_offsets, *idx_offsets;
    uint64_t vertex_offset, max_index;  // max_index: per path, ~0 for none
    uint32_t* words;                    // [0] scan error, [1] failed paths
    uint64_t* host;                     // totals, the words above, STROKE_VERBS_READ words
};
// Counts of every path (vtx_counts, idx_counts, status of `a`), the paths in walk_list apart.
// `verbs_hint`: about how many verbs the batch has (sizes the grids, and with `finish`, which may be
// null, chooses who sums the verbs). finish: for STROKE_FINISH_PATHS paths at most.
cudaError_t launch_stroke_verbs_count(const StrokeArgs& a, const StrokeVerbs& v,
                                      uint32_t verbs_hint, int num_sms, const SideStreams& side,
                                      const StrokeFinish* finish, cudaStream_t s);
// The stepper's part of it (stroke_steps.cu): counts of a variable-width stroke once the kept points
// are known, and the output of variable widths, vertex sources and attribute records.
void launch_stroke_steps_count(const StrokeArgs& a, const StrokeVerbs& v, uint32_t verbs_hint,
                               int num_sms, const SideStreams& side, cudaStream_t s);
// Records: advancements beside the count for up to this many paths, before the emit kernels for more,
// where they would keep SMs from the count (1,000 paths of 16 cubics 306 -> 261 us, 10,000 646 ->
// 562, but 20,000 curve paths 2486 -> 2615).
constexpr uint32_t STROKE_ADVANCE_EARLY = 12288;
void launch_stroke_advance(const StrokeArgs& a, const StrokeVerbs& v, int num_sms,
                           const SideStreams& side, cudaStream_t s);
void join_stroke_advance(const SideStreams& side, cudaStream_t s);
cudaError_t launch_stroke_steps_emit(const StrokeArgs& a, const StrokeVerbs& v,
                                     uint32_t verbs_hint, int num_sms, const SideStreams& side,
                                     cudaStream_t s);
// Output of the paths that launch_stroke_verbs_count counted. `runs`: words[3].
cudaError_t launch_stroke_verbs_emit(const StrokeArgs& a, const StrokeVerbs& v,
                                     uint32_t verbs_hint, bool runs, int num_sms,
                                     const SideStreams& side, cudaStream_t s);

}  // namespace lg
