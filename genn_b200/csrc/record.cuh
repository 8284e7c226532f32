// Spike recordings on their way to the host.
//
// A recording is one bit per neuron and time step ([step][batch][32-neuron word], neuron_update.cuh) and almost all
// zeros at cortical rates, so the device lists the non-zero words of all recorded populations as (index, word) pairs
// and only those travel.  The list comes in the order of the arrays: a block counts its chunk, a second kernel places
// it behind the chunks before, so that the host decodes spikes with one pass over the pairs instead of one over
// every bit (Runtime::getRecordedEvents, runtime.cc:855-913, walks them all).  Two launches for all populations;
// the words are read twice, the second time from L2 (0.97 MB for 100 steps of the 77 169-neuron microcircuit).
// Measured with its 1 650 spikes: pull and decode 0.2 ms, 20 ms while the host unpacked every bit of the recording.
#pragma once

#include <string.h>

#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace b200
{
constexpr unsigned int RECORD_BLOCK = 256;
constexpr unsigned int RECORD_WORDS = 16;                                   // consecutive words of a thread
constexpr unsigned int RECORD_CHUNK = RECORD_BLOCK * RECORD_WORDS;          // words of a block
constexpr unsigned int RECORD_ARRAYS = 48;                                  // arrays of one launch

struct RecordArrays
{
    const unsigned int *words[RECORD_ARRAYS];
    unsigned int num_words[RECORD_ARRAYS];
    unsigned int base[RECORD_ARRAYS];               // index of the array's first word in the list
    unsigned int chunk_start[RECORD_ARRAYS + 1];    // chunks of this launch before each array
    unsigned int num;
    unsigned int first_chunk;                       // chunks of earlier launches
};

// What precedes the pairs in the list: filled in by the last chunk.
struct RecordHeader
{
    unsigned int count;         // non-zero words, those beyond the list's capacity included
    unsigned int error;         // StepState::error
};

struct RecordSlice
{
    unsigned int array, first;      // which array, first word of this thread in it
    unsigned int n;                 // words of this thread (0 .. RECORD_WORDS)
};

__device__ __forceinline__ RecordSlice recordSlice(const RecordArrays &A)
{
    RecordSlice s;
    s.array = findGroup(A.chunk_start, A.num, blockIdx.x);
    s.first = (blockIdx.x - A.chunk_start[s.array]) * RECORD_CHUNK + threadIdx.x * RECORD_WORDS;
    const unsigned int total = A.num_words[s.array];
    s.n = (s.first < total) ? min(RECORD_WORDS, total - s.first) : 0u;
    return s;
}

// (array starts are 256-byte aligned: a full slice is four aligned 16-byte loads)
__device__ __forceinline__ unsigned int recordLoad(const RecordArrays &A, const RecordSlice &s, unsigned int (&w)[RECORD_WORDS])
{
    const unsigned int *p = A.words[s.array] + s.first;
    #pragma unroll
    for(unsigned int i = 0; i < RECORD_WORDS; i += 4) {
        if(i + 4u <= s.n) {
            const uint4 v = *reinterpret_cast<const uint4*>(p + i);
            w[i] = v.x; w[i + 1] = v.y; w[i + 2] = v.z; w[i + 3] = v.w;
        }
        else {
            #pragma unroll
            for(unsigned int j = 0; j < 4; j++) w[i + j] = (i + j < s.n) ? p[i + j] : 0u;
        }
    }
    unsigned int c = 0;
    #pragma unroll
    for(unsigned int i = 0; i < RECORD_WORDS; i++) c += w[i] ? 1u : 0u;
    return c;
}

__device__ __forceinline__ unsigned int recordBlockSum(unsigned int v, unsigned int *warpSums)
{
    v = __reduce_add_sync(0xFFFFFFFFu, v);
    if((threadIdx.x & 31u) == 0) warpSums[threadIdx.x >> 5] = v;
    __syncthreads();
    unsigned int sum = 0;
    #pragma unroll
    for(unsigned int i = 0; i < RECORD_BLOCK / 32; i++) sum += warpSums[i];
    return sum;
}

__global__ void __launch_bounds__(RECORD_BLOCK)
recordCountKernel(const RecordArrays A, unsigned int *counts)
{
    __shared__ unsigned int warpSums[RECORD_BLOCK / 32];
    unsigned int w[RECORD_WORDS];
    const unsigned int sum = recordBlockSum(recordLoad(A, recordSlice(A), w), warpSums);
    if(threadIdx.x == 0) counts[A.first_chunk + blockIdx.x] = sum;
}

__global__ void __launch_bounds__(RECORD_BLOCK)
recordListKernel(const RecordArrays A, const unsigned int *counts, unsigned int num_chunks, RecordHeader *header,
                 uint2 *pairs, unsigned int capacity, const StepState *state)
{
    __shared__ unsigned int warpSums[RECORD_BLOCK / 32], warpCounts[RECORD_BLOCK / 32];
    const unsigned int me = A.first_chunk + blockIdx.x;
    unsigned int before = 0;
    for(unsigned int i = threadIdx.x; i < me; i += RECORD_BLOCK) before += counts[i];
    before = recordBlockSum(before, warpSums);
    const RecordSlice s = recordSlice(A);
    unsigned int w[RECORD_WORDS];
    const unsigned int mine = recordLoad(A, s, w);
    // position of this thread's first pair inside the chunk
    const unsigned int lane = threadIdx.x & 31u;
    unsigned int incl = mine;
    #pragma unroll
    for(int o = 1; o < 32; o <<= 1) {
        const unsigned int v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if(lane >= (unsigned int)o) incl += v;
    }
    if(lane == 31u) warpCounts[threadIdx.x >> 5] = incl;
    __syncthreads();
    unsigned int at = before + incl - mine;
    for(unsigned int i = 0; i < (threadIdx.x >> 5); i++) at += warpCounts[i];
    #pragma unroll
    for(unsigned int i = 0; i < RECORD_WORDS; i++) {
        if(w[i]) {
            if(at < capacity) pairs[at] = make_uint2(A.base[s.array] + s.first + i, w[i]);
            at++;
        }
    }
    if(me == num_chunks - 1u && threadIdx.x == RECORD_BLOCK - 1u) {
        header->count = at;             // the last thread of the last chunk
        header->error = state->error;
    }
}

// Set bits of `n` words (with the processor's own instruction where it has one: the portable count takes as long as the rest
// of the decoding).
__attribute__((target("popcnt"))) inline uint64_t countBitsNative(const uint32_t *words, uint64_t n)
{
    uint64_t bits = 0, i = 0;
    for(; i + 2u <= n; i += 2u) {
        uint64_t two;
        memcpy(&two, words + i, sizeof(two));
        bits += (uint64_t)__builtin_popcountll(two);
    }
    if(i < n) bits += (uint64_t)__builtin_popcount(words[i]);
    return bits;
}
inline uint64_t countBits(const uint32_t *words, uint64_t n)
{
    static const bool native = __builtin_cpu_supports("popcnt");
    if(native) return countBitsNative(words, n);
    uint64_t bits = 0;
    for(uint64_t i = 0; i < n; i++) bits += (uint64_t)__builtin_popcount(words[i]);
    return bits;
}

// Pairs [from, to) of a list, all from one turn of the ring.  The list is in index order, so the row and the batch entry of a pair are
// those of the one before or come soon after (divisions took half of the time).
struct RecordPairs
{
    const uint32_t *pairs;
    uint32_t base, rows, batch, words_per_row, first_row, first_id, lastMask;
    double start, dt;
    uint64_t *counts;
    double *const *times;
    uint32_t *const *ids;
};

__attribute__((always_inline)) inline void decodePairsAs(const RecordPairs &R, uint64_t from, uint64_t to)
{
    if(from >= to) return;
    const uint32_t words = R.words_per_row, first = R.pairs[2 * from] - R.base;
    // section: one batch entry of one row
    uint64_t section = first / words, sectionEnd = (section + 1u) * words;
    uint32_t row = (uint32_t)(section / R.batch), b = (uint32_t)(section - (uint64_t)row * R.batch);
    auto timeOf = [&] { return R.start + (double)(row >= R.first_row ? row - R.first_row : row + R.rows - R.first_row) * R.dt; };
    double t = timeOf();
    uint64_t at = R.counts[b];
    // (an entry that has nothing but padding may come without arrays)
    const bool store = R.ids != nullptr;
    double *times = store ? R.times[b] : nullptr;
    uint32_t *ids = store ? R.ids[b] : nullptr;
    for(uint64_t i = from; i < to; i++) {
        const uint32_t index = R.pairs[2 * i] - R.base;
        uint32_t word = R.pairs[2 * i + 1];
        if(index >= sectionEnd) {
            R.counts[b] = at;
            do {
                sectionEnd += words;
                if(++b == R.batch) {
                    b = 0;
                    row++;
                }
            } while(index >= sectionEnd);
            t = timeOf();
            at = R.counts[b];
            if(store) {
                times = R.times[b];
                ids = R.ids[b];
            }
        }
        if(index + 1u == sectionEnd) word &= R.lastMask;
        if(!store) {
            at += (uint64_t)__builtin_popcount(word);
            continue;
        }
        const uint32_t id = R.first_id + (uint32_t)(index - (sectionEnd - words)) * 32u;
        for(; word; word &= word - 1u, at++) {
            times[at] = t;
            ids[at] = id + (uint32_t)__builtin_ctz(word);
        }
    }
    R.counts[b] = at;
}
__attribute__((target("popcnt,bmi"))) inline void decodePairsNative(const RecordPairs &R, uint64_t from, uint64_t to) { decodePairsAs(R, from, to); }

// Host side.  The spikes in a recording of one population: bits of `words` ([rows][batch][words_per_row], the whole
// array) or, if `words` is NULL, of the (index, word) pairs of a list in index order in which the array begins at
// index `base`.  Row `first_row` is the oldest (the recording is a ring over the steps).  Without `ids`, counts them per
// batch entry; with it, stores time (start + row * dt, rows counted from the oldest) and neuron id of every spike,
// ordered by time, then id.  Bits at or beyond `num_neurons` are padding.
inline void decodeRecording(const uint32_t *words, const uint32_t *pairs, uint64_t num_pairs, uint32_t base, uint32_t rows,
                            uint32_t batch, uint32_t words_per_row, uint32_t first_row, uint32_t num_neurons, uint32_t first_id,
                            double start, double dt, uint64_t *counts, double *const *times, uint32_t *const *ids)
{
    for(uint32_t b = 0; b < batch; b++) counts[b] = 0;
    const uint32_t perRow = batch * words_per_row;
    const uint32_t lastMask = (num_neurons & 31u) ? (1u << (num_neurons & 31u)) - 1u : 0xFFFFFFFFu;
    auto take = [&](uint32_t row, uint32_t b, uint32_t w, uint32_t word) {
        if(w + 1u == words_per_row) word &= lastMask;
        if(!ids) {
            counts[b] += (uint64_t)__builtin_popcount(word);
            return;
        }
        uint64_t at = counts[b];
        const double t = start + (double)(row >= first_row ? row - first_row : row + rows - first_row) * dt;
        for(; word; word &= word - 1u, at++) {
            times[b][at] = t;
            ids[b][at] = first_id + w * 32u + (uint32_t)__builtin_ctz(word);
        }
        counts[b] = at;
    };
    if(words) {
        for(uint32_t i = 0; i < rows; i++) {
            const uint32_t row = (first_row + i < rows) ? first_row + i : first_row + i - rows;
            const uint32_t *r = words + (uint64_t)row * perRow;
            for(uint32_t b = 0; b < batch; b++) {
                const uint32_t *const mine = r + b * words_per_row;
                if(!ids) {
                    counts[b] += countBits(mine, words_per_row - 1u) + (uint64_t)__builtin_popcount(mine[words_per_row - 1u] & lastMask);
                    continue;
                }
                // two words at a time: most are zero
                uint32_t w = 0;
                for(; w + 2u <= words_per_row; w += 2u) {
                    uint64_t two;
                    memcpy(&two, mine + w, sizeof(two));
                    if(!two) continue;
                    if(mine[w]) take(row, b, w, mine[w]);
                    if(mine[w + 1u]) take(row, b, w + 1u, mine[w + 1u]);
                }
                if(w < words_per_row && mine[w]) take(row, b, w, mine[w]);
            }
        }
        return;
    }
    auto find = [&](uint64_t index) {       // first pair at or behind `index`
        uint64_t lo = 0, hi = num_pairs;
        while(lo < hi) {
            const uint64_t m = (lo + hi) / 2;
            if(pairs[2 * m] < index) lo = m + 1; else hi = m;
        }
        return lo;
    };
    const uint64_t begin = find(base), split = find((uint64_t)base + (uint64_t)first_row * perRow);
    const uint64_t end = find((uint64_t)base + (uint64_t)rows * perRow);
    const RecordPairs R{pairs, base, rows, batch, words_per_row, first_row, first_id, lastMask, start, dt, counts, times, ids};
    static const bool native = __builtin_cpu_supports("popcnt") && __builtin_cpu_supports("bmi");
    const uint64_t part[2][2] = {{split, end}, {begin, split}};
    for(const auto &p : part) {
        if(native) decodePairsNative(R, p[0], p[1]);
        else decodePairsAs(R, p[0], p[1]);
    }
}
}   // namespace b200
