// lyap_args.h -- kernel parameter block of the lambda kernels (plain types only: also compiled at run time).
#pragma once

namespace lyap {

// Per-step parameter selectors, 2 bits per step (0 = A/column, 1 = B/row, 2 = C/scalar), 16 steps per
// 32-bit word.  Warm-up steps start at word 0, accumulation steps at word `acc_word0`, each region in
// its own words so both can be walked in whole 16-step chunks plus one partial chunk.  A region longer than
// its share of the table stores one period of the sequence in whole words (lcm(len, 16) steps) and repeats
// it: word w of a region is sel[word0 + w % wrap].
constexpr int kStepsPerWord = 16;
// Most steps between two exit tests of the exact kernels.
constexpr int kMaxChunk = 80;
// Steps that have to be left for the exact kernels' turning to an orbit's cycle to pay.
constexpr int kLeastLeft = 160;
// The fast kernels' chunk for a sequence whose pairs of steps repeat every `bs` steps: blocks of whole periods and at least 16
// steps, so many of them that cycles of two, three, four and eight periods go into a chunk as far as 130 steps can hold them.
// An exit test costs more the shorter the chunk is, a cycle is found the later the longer it is: 4096^2 of "AABAB" 200 + 2000
// in chunks of 80 / 120 / 160 steps 3.42 / 3.39 / 3.47 ms (fp32), 6.44 / 6.28 / 6.51 (fp64, 4 pixels a thread).
__host__ __device__ constexpr int fast_block_periods(int bs) { return (kStepsPerWord + bs - 1) / bs; }
__host__ __device__ constexpr int fast_chunk_blocks(int bs) { return bs * fast_block_periods(bs) <= 20 && bs != 6 ? 6 : 4; }
__host__ __device__ constexpr int fast_chunk(int bs) { return bs * fast_block_periods(bs) * fast_chunk_blocks(bs); }
// Steps after which a turn of a cycle is looked at: whole periods, and some where they are short (a chunk is a multiple of it).
__host__ __device__ constexpr int fast_unit(int bs) { return bs <= 4 ? 8 : bs; }
constexpr int kMaxSelWords = 896;  // 14336 distinct steps through kernel parameters (kernel parameter space is 4 KB)

struct LambdaArgs {
    double min_x, min_y, dx, dy, c_value;
    long long row_begin;   // global index of the first row of this launch
    long long n_pixels;    // rows * width
    long long wide_tiles;  // exact kernel: warp-tiles of several pixels a thread, before the rest goes in tiles of one
    int width;
    int warmup, iterations;
    int acc_word0;
    int fast_ok_c;         // c_value is positive, finite and of ordinary magnitude (or unused)
    int wu_wrap, acc_wrap; // words after which each region's selectors repeat (>= the region's words when it is stored whole)
    int acc_period;        // steps after which the accumulation's selectors repeat (a fast mode's are whole units), 0 when that is more than kMaxChunk
    int acc_chunk;         // steps between two exit tests of the generic kernels: a multiple of acc_period, if there is one
    unsigned* queue;       // exact kernel: tiles handed out so far and warps that are done, both zero between launches; null: no queue
    unsigned long long* cycle_steps;   // counts steps taken from an orbit's cycle instead of being walked (may be null)
    unsigned int sel[kMaxSelWords];
};

}  // namespace lyap
