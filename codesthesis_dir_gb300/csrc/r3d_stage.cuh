// Shared memory of the 3D solves' line phases (r3d.cu): how many lines a chunk
// stages and what they take.  The device forms chunks by this rule and the host
// forms the groups of lines that must share one.
#pragma once

#include "warpline.cuh"

#define R3_THREADS 256
// The staged right-hand sides and, behind them, their factors.
#define R3_CHUNK_BYTES (44 * 1024)
#define R3_FAC_BYTES (52 * 1024)
// The longest FP64 line: one that reaches beyond the first area lies over the
// factors' too, which a line of that length does not stage (7 n doubles).
#define R3_MAX_ROWS ((R3_CHUNK_BYTES + R3_FAC_BYTES) / 8)

// Elements that nl staged lines of n rows take: FP64 [row][line] with an odd
// pitch (no bank conflicts when each thread walks its line), FP32 [line][row],
// padded per lane (warpline.cuh).
__host__ __device__ __forceinline__ int r3_stage_words(bool f64, int n, int nl) { return f64 ? n * (nl | 1) : nl * wl_pitch(n); }

// Lines of n rows that a chunk of direction dir holds at most, their tables len
// elements each; fewer lines take no more room.
__host__ __device__ __forceinline__ int r3_chunk(bool f64, int dir, int n, int len)
{
    const int words = R3_CHUNK_BYTES / (f64 ? 8 : 4), line = f64 ? n : wl_pitch(n);
    int c = R3_THREADS < words / line ? R3_THREADS : words / line;
    if (f64 && r3_stage_words(true, n, c) > words) --c;   // an even number has the pitch of the next odd one
    if (!f64 && dir == 1) {                               // a table per line
        const int tables = R3_FAC_BYTES / 4 / len;
        c = c < tables ? c : tables;
    }
    return c > 1 ? c : 1;
}
