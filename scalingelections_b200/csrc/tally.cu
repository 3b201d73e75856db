// Ballot tally on sm_100a: build_pairwise_preferences (scaling_elections.py:51-88) redesigned.
//
// The reference scatters d[r[a]][r[b]] += 1 for every ordered pair of every ballot (py:46-48),
// one voter at a time. Here the tally is a reduction over voters of a comparison:
//   d[i][j] = #{v : pos_v(i) < pos_v(j)}
// where pos_v is ballot v's rank position of each candidate after the reference's completion
// rule (missing ids appended in ascending order, py:75-83). Every completed ballot is a
// permutation, so for i != j exactly one of (i above j), (j above i) holds and
// d[j][i] = V - d[i][j]: only the upper-triangle tiles are computed.
//
// Kernel 1 (positions_kernel) writes pos as f32 [V][Cq] (exact integers), validating ids
// (range, repeats). Kernel 2 (pack_planes_kernel) packs each 32-voter chunk into bit planes.
//
// A ballot that names a candidate more than once is not a permutation, and the reference
// counts it pair by pair all the same (py:46-48; py:75 completes it only when its length
// differs from C). Such an "irregular" ballot gets place 0 for every candidate, so the
// bit-sliced count sees no pair for it in either direction, and it is left out of the
// complement V - d[i][j]. irregular_kernel then adds its pairs exactly as the reference does,
// diagonal included, with atomics.
// For C < 2048, places_planes_kernel does both in one pass and keeps the places in shared
// memory. Kernel 3 (count_bits_kernel, one CTA per SM) streams the planes of each upper tile's two
// 128-candidate strips into shared memory with TMA and counts per 8 x 4 register micro-tile
// with a bit-serial borrow chain (one lop3 per plane) and a popc per 32 voters.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "common.cuh"
#include "positions.cuh"

namespace se {
namespace closure {
se_status_t make_map(CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer, uint64_t pitch_bytes,
                     uint32_t box_x, uint32_t box_y);
}

namespace tally {

constexpr int kTile = 128;     // candidates per tile edge
constexpr int kVC = 32;        // voters per TMA chunk
constexpr int kThreads = 512;  // 8 x 4 cells per thread
constexpr uint32_t kErrRange = 2;
constexpr uint32_t kErrTimeout = 1;
constexpr uint32_t kErrOffsets = 8;  // replaces any other code
constexpr uint32_t kMaxPolls = 1u << 26;

int64_t padded(int C) { return round_up(C, kTile); }

// Irregular ballots (a repeated id) of one call, in the workspace after the error word:
// a count, the number per 32-voter chunk (the count kernel leaves them out of V - d[i][j]) and
// the list of their ballot indices (for irregular_kernel).
struct Irregular {
    uint32_t* n;         // irregular ballots recorded
    uint32_t* chunk;     // [ceil(V / 32)]: irregular ballots per 32-voter chunk
    uint32_t* list;      // [V]: their ballot indices, in no particular order
};

__device__ __forceinline__ void record_irregular(const Irregular& irr, int64_t v) {
    irr.list[atomicAdd(irr.n, 1u)] = uint32_t(v);
    atomicAdd(irr.chunk + v / 32, 1u);
}

// Ballot v's span of ids. With num_ids >= 0 the offsets are checked as they are read: they must
// start at 0, never decrease and end at num_ids. A ballot whose span breaks that is reported and
// read as empty, so no kernel follows a bad bound, and the kernels after the one that reads the
// offsets leave the output alone; the check costs the tally no pass of its own.
struct Span {
    int64_t beg, len;
    bool ok;
};
__device__ __forceinline__ Span ballot_span(const int64_t* offsets, int64_t id_base, int64_t v, int64_t V, int C,
                                            int64_t num_ids) {
    if (!offsets) return {v * C, C, true};
    const int64_t beg = offsets[v] - id_base, end = offsets[v + 1] - id_base;
    if (num_ids >= 0 && (beg < 0 || end < beg || end > num_ids || (v == 0 && beg != 0) || (v == V - 1 && end != num_ids)))
        return {0, 0, false};
    return {beg, end - beg, true};
}

// ------------------------------------------------------------------------------------------
// Positions (from C = 2048 on; below that places_planes_kernel keeps them on the SM):
// pos[v][c] = place of candidate c on completed ballot v, one CTA per ballot, the row built in
// shared memory up to C = 23552 (block_places_u16 in positions.cuh) and in global memory
// beyond (block_positions). Id is int32_t, or uint16_t / uint8_t for packed ballots.
// Ballot v is ids[offsets[v] - id_base, offsets[v + 1] - id_base), or ids[v * C, (v + 1) * C)
// when offsets is null (complete ballots).
// ------------------------------------------------------------------------------------------
constexpr int kPosThreads = 256;

// 16-bit place rows up to 46 KiB of dynamic shared memory: with the kernel's static shared
// memory that stays within the 48 KiB a block gets without raising its limit.
constexpr int kPosRowMaxCq = 23552;

// ROW: the place row is built in shared memory (block_places_u16, Cq halfwords of dynamic
// shared memory) and written out coalesced; else in global memory (block_positions).
template <typename Id, bool ROW>
__global__ void __launch_bounds__(kPosThreads)
    positions_kernel(const Id* __restrict__ ids, const int64_t* __restrict__ offsets, int64_t id_base, int64_t V,
                     int C, int64_t Cq, float* __restrict__ pos, Irregular irr, int64_t num_ids,
                 uint32_t* __restrict__ err) {
    extern __shared__ __align__(16) uint16_t row[];
    const int64_t v = blockIdx.x;
    const Span span = ballot_span(offsets, id_base, v, V, C, num_ids);
    const int64_t beg = span.beg, len = span.len;
    if (!span.ok && threadIdx.x == 0) atomicExch(err, kErrOffsets);
    __shared__ int scratch[33];
    int code;
    if constexpr (ROW) code = block_places_u16(ids + beg, len, C, int(Cq), row, pos + v * Cq, scratch);
    else code = block_positions(ids + beg, len, C, Cq, pos + v * Cq, scratch);
    if (code == kPosRepeat) {  // every thread got the same code after the block-wide check
        for (int64_t c = threadIdx.x; c < Cq; c += blockDim.x) pos[v * Cq + c] = 0.0f;
        if (threadIdx.x == 0) record_irregular(irr, v);
    } else if (code != kPosOk && threadIdx.x == 0) {
        raise_device_error(err, uint32_t(code));
    }
}

template <typename Id>
void launch_positions(const Id* ids, const int64_t* offsets, int64_t id_base, int64_t V, int C, int64_t Cq,
                      float* pos, const Irregular& irr, int64_t num_ids, uint32_t* err, cudaStream_t s) {
    if (Cq <= kPosRowMaxCq)
        positions_kernel<Id, true><<<unsigned(V), kPosThreads, size_t(Cq) * 2, s>>>(ids, offsets, id_base, V, C, Cq,
                                                                                 pos, irr, num_ids, err);
    else
        positions_kernel<Id, false><<<unsigned(V), kPosThreads, 0, s>>>(ids, offsets, id_base, V, C, Cq, pos, irr,
                                                                        num_ids, err);
}

// ------------------------------------------------------------------------------------------
// Bit-sliced counting. For a chunk of 32 voters, bit k of every voter's place of candidate c is
// gathered into one word: plane[ch][k][c] (bit v = bit k of pos_{32 ch + v}(c)). Then
// pos(i) < pos(j) for all 32 voters at once is the borrow out of the bit-serial subtraction
// pos(i) - pos(j): borrow' = MAJ(~a_k, b_k, borrow) over the planes from the least significant,
// one `lop3.b32` (LUT 0x8E) per plane, and one `popc` adds the 32 answers. With B = bits of
// C - 1 planes that is about (B + 2) / 32 ALU instructions per voter pair, against two FP32
// instructions in the direct form.
// ------------------------------------------------------------------------------------------
constexpr int kBitStages = 4;

// Bit planes of 16 bits of 32 voters' places. On entry w[u] holds voter u's bits in its low half
// and voter u + 16's in its high half; on return bit v of w[k] is bit k of voter v. Both halves
// are transposed at once by swapping off-diagonal squares of 8, 4, 2 and 1 bits: about 130
// instructions a word of 32 places (the rows past the last plane are dead code), against two per
// voter and plane (640 at B = 10) when each bit is extracted and inserted by itself. With half the
// registers places_planes_kernel also runs two CTAs per SM: 174 -> 116 us for 60000 ragged ballots
// at C = 1000; pack_planes_kernel 35 -> 26 us at C = V = 4096.
__device__ __forceinline__ void transpose_places(uint32_t (&w)[16]) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const uint32_t a = w[u], b = w[u + 8];
        w[u] = __byte_perm(a, b, 0x6240);
        w[u + 8] = __byte_perm(a, b, 0x7351);
    }
#pragma unroll
    for (int d = 4; d >= 1; d >>= 1) {
        const uint32_t m = d == 4 ? 0x0F0F0F0Fu : d == 2 ? 0x33333333u : 0x55555555u;
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            if (u & d) continue;
            const uint32_t a = w[u], b = w[u + d];
            w[u] = (a & m) | ((b << d) & ~m);
            w[u + d] = ((a >> d) & m) | (b & ~m);
        }
    }
}

// planes[(ch * B + k) * Cq + c] for the chunks of voters [0, V); voters past V count as place 0.
// B is a template parameter so that only B planes of bit work are done, in registers.
template <int B>
__global__ void __launch_bounds__(256)
    pack_planes_kernel(const float* __restrict__ pos, int64_t V, int64_t Cq, uint32_t* __restrict__ planes) {
    const int64_t c = int64_t(blockIdx.y) * blockDim.x + threadIdx.x;  // grid: (chunks, ceil(Cq / 256))
    const int64_t ch = blockIdx.x;
    if (c >= Cq) return;
    uint32_t p[32];
#pragma unroll
    for (int v = 0; v < 32; ++v) {
        const int64_t voter = ch * 32 + v;
        p[v] = voter < V ? uint32_t(pos[voter * Cq + c]) : 0u;
    }
#pragma unroll
    for (int k0 = 0; k0 < B; k0 += 16) {
        uint32_t w[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) w[u] = __byte_perm(p[u], p[u + 16], k0 ? 0x7632 : 0x5410);
        transpose_places(w);
#pragma unroll
        for (int k = 0; k < 16; ++k)
            if (k0 + k < B) planes[(ch * B + k0 + k) * Cq + c] = w[k];
    }
}

// Places and planes in one pass, for C < 2048: one CTA of 32 warps per 32-ballot chunk. Warp
// w writes the places of ballot 32 ch + w as 16-bit values into row w of shared memory. Then
// each thread takes one candidate: it reads the candidate's 32 places down the column (lanes
// read neighbouring halfwords of one row, no bank conflicts) and builds each plane word in
// registers. The places never leave the SM.
constexpr int kFusedMaxCq = 2048;
inline size_t fused_smem(int64_t Cq) { return size_t(32) * size_t(Cq + 2) * 2; }

template <typename Id, int B>
__global__ void __launch_bounds__(1024, 2)
    places_planes_kernel(const Id* __restrict__ ids, const int64_t* __restrict__ offsets, int64_t id_base,
                         int64_t V, int C, int Cq, uint32_t* __restrict__ planes, Irregular irr, int64_t num_ids,
                         uint32_t* __restrict__ err) {
    extern __shared__ __align__(16) uint16_t rows[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pitch = Cq + 2;  // halfwords; rows start 4 bytes apart modulo 128
    const int64_t ch = blockIdx.x;
    const int64_t v = ch * 32 + warp;
    uint16_t* row = rows + warp * pitch;
    if (v < V) {
        const Span span = ballot_span(offsets, id_base, v, V, C, num_ids);
        if (!span.ok && lane == 0) atomicExch(err, kErrOffsets);
        const int code = warp_places_u16(ids + span.beg, span.len, C, Cq, row);
        if (code == kPosRepeat) {  // an irregular ballot: place 0 everywhere, counted apart
            __syncwarp();
            for (int c = lane; c < Cq; c += 32) row[c] = 0;
            if (lane == 0) record_irregular(irr, v);
        } else if (code != kPosOk && lane == 0) {
            raise_device_error(err, uint32_t(code));
        }
    } else {
        for (int c = lane; c < Cq; c += 32) row[c] = 0;  // voters past V count as place 0
    }
    __syncthreads();
    for (int c = threadIdx.x; c < Cq; c += blockDim.x) {
        uint32_t w[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) w[u] = rows[u * pitch + c] | uint32_t(rows[(u + 16) * pitch + c]) << 16;
        transpose_places(w);
#pragma unroll
        for (int k = 0; k < B; ++k) planes[(ch * B + k) * int64_t(Cq) + c] = w[k];
    }
}

__device__ __forceinline__ uint32_t borrow_step(uint32_t a, uint32_t b, uint32_t br) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0x8E;" : "=r"(r) : "r"(a), "r"(b), "r"(br));
    return r;
}

inline size_t bits_smem(int B) { return size_t(kBitStages) * 2 * B * kTile * 4 + kBitStages * 8; }

// How the count's CTAs share the work. The tiles are ordered with the n1 = R (R - 1) / 2 tiles
// above the diagonal first, row by row, then the R diagonal tiles. CTA b of the G (one per SM)
// takes the whole tiles b, b + G, .. of the first `rounds` * G, all above the diagonal. The rest
// is laid end to end as a line of (tile, 32-voter chunk) units and cut into G equal ranges, where
// a unit above the diagonal weighs 5 and a diagonal one 4 (count_bits_kernel leaves out warps
// there). se_tally, us, with weights 1 : 1 / 4 : 3 / 5 : 4 / 6 : 5: C = 256, V = 100000 212 / 208 /
// 205 / 211; C = 500, V = 100000 508 / 483 / 484 / 489; C = 1000, V = 60000 914 / 912 / 886 / 894; C =
// 1500, V = 30000 1028 / 1052 / 1006 / 1017; C = 2000, V = 20000 1224 / 1273 / 1212 / 1214; C = 3000,
// V = 8000 1192 / 1190 / 1181 / 1166; 1 % or less between them from C = 4096 on. A range ends anywhere
// inside a tile; such a tile's counts arrive as atomic adds. `whole` moves the ends to tile ends. So
// no SM waits for a last partial wave, and a CTA has at most two split tiles to add, however many
// voters there are.
struct CountSplit {
    int64_t rounds;
    bool whole;
};

__host__ __device__ inline int64_t tiles_above(int R) { return int64_t(R) * (R - 1) / 2; }

// Tile t of that order.
__device__ __forceinline__ void count_tile(int64_t t, int R, int& I, int& J) {
    const int64_t n1 = tiles_above(R);
    if (t < n1) {
        upper_pair(t, R - 1, I, J);
        ++J;
    } else {
        I = J = int(t - n1);
    }
}

// First unit of CTA b's range of the line (b = G: its end).
__device__ __forceinline__ int64_t range_start(const CountSplit& sp, int R, int64_t chunks, int64_t b, int64_t G) {
    const int64_t above = tiles_above(R) - sp.rounds * G;  // tiles of the line above the diagonal
    if (b == 0) return 0;
    if (b == G) return (above + R) * chunks;
    if (sp.whole) return (above + R) * b / G * chunks;
    const int64_t x = (5 * above + 4 * R) * chunks * b / G;
    return x <= 5 * above * chunks ? x / 5 : above * chunks + (x - 5 * above * chunks) / 4;
}

// Zeroes the tiles that range ends cut, and their mirrors: blocks (b, *) look at the start of range
// b + 1 of G = gridDim.x + 1, and leave a tile that an earlier range's start cuts to that one's.
// Each of the gridDim.y blocks of a tile takes its share of the rows.
constexpr int kZeroParts = 8;

__global__ void __launch_bounds__(256)
    zero_tiles_kernel(uint32_t* __restrict__ out, int64_t ld_out, int C, int R, int64_t chunks, CountSplit sp,
                      const uint32_t* __restrict__ err) {
    if (*err == kErrOffsets) return;
    const int64_t b = int64_t(blockIdx.x) + 1, G = int64_t(gridDim.x) + 1;
    const int64_t u = range_start(sp, R, chunks, b, G), t = u / chunks;
    if (u % chunks == 0) return;
    const int64_t before = range_start(sp, R, chunks, b - 1, G);
    if (before / chunks == t && before % chunks != 0) return;
    int I, J;
    count_tile(sp.rounds * G + t, R, I, J);
    for (int e = blockIdx.y * 256 + threadIdx.x; e < kTile * kTile; e += gridDim.y * 256) {
        const int r = e / kTile, c = e % kTile;
        if (I * kTile + r < C && J * kTile + c < C) out[int64_t(I * kTile + r) * ld_out + J * kTile + c] = 0u;
        if (I != J && J * kTile + r < C && I * kTile + c < C) out[int64_t(J * kTile + r) * ld_out + I * kTile + c] = 0u;
    }
}

// Counting over upper tiles (I <= J): d[I][J] and, for I < J, d[J][I] = V - d[I][J]. One CTA per
// SM works through its tiles (CountSplit): the two 128-candidate plane strips of each 32-voter
// chunk are staged by TMA (box {128, B}) through a 4-stage ring that runs on across its tiles, so
// the next tile's first chunks arrive while this one's counts go out. The ALU pipe is the bound
// (83 % active at C = V = 4096, 919 us; the warps wait for that pipe or for a turn to issue). Before the
// tiles were shared out evenly, each CTA took one tile or a fixed share of one, and the last wave, the
// many small shares' adds and the full diagonal tiles cost the rest.
// A diagonal tile's mirror image lies in itself: its 6 warps (of 16, one 32 x 32 block each) below
// the diagonal count nothing, and the warps above write both cells. The blocks are dealt to the
// warps such that each scheduler (warp mod 4) keeps at most 3 of its 4.
// B (the planes per chunk) is a template parameter: the plane loop unrolls fully.
template <int B>
__global__ void __launch_bounds__(kThreads, 1)
    count_bits_kernel(const __grid_constant__ CUtensorMap mapPl, int64_t V, int C, int R, CountSplit sp,
                      uint32_t* __restrict__ out, int64_t ld_out, bool accumulate,
                      const uint32_t* __restrict__ irr_chunk, uint32_t* __restrict__ err) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint32_t* sI = reinterpret_cast<uint32_t*>(smem_raw);  // [kBitStages][B][kTile]
    uint32_t* sJ = sI + kBitStages * B * kTile;            // [kBitStages][B][kTile]
    uint64_t* bars = reinterpret_cast<uint64_t*>(sJ + kBitStages * B * kTile);
    constexpr uint32_t stage_words = uint32_t(B) * kTile;
    constexpr uint32_t stage_bytes = 2u * stage_words * 4u;

    const int64_t G = gridDim.x, cta = blockIdx.x;
    const int chunks = int((V + kVC - 1) / kVC);
    const int64_t start = range_start(sp, R, chunks, cta, G);
    const int64_t in_rounds = sp.rounds * chunks;  // units in whole-tile rounds
    // None where an earlier kernel has refused the offsets (this one only replaces a 0 in err).
    const int64_t units = *err == kErrOffsets ? 0 : in_rounds + range_start(sp, R, chunks, cta + 1, G) - start;
    // Unit n of this CTA: its tile and chunk.
    auto locate = [&](int64_t n, int& I, int& J, int& ch) {
        const int64_t u = n < in_rounds ? n : start + (n - in_rounds);
        const int64_t q = u / chunks;
        ch = int(u - q * chunks);
        count_tile(n < in_rounds ? cta + G * q : sp.rounds * G + q, R, I, J);
    };
    auto load = [&](int s, int I, int J, int ch) {
        mbar_arrive_expect_tx(&bars[s], stage_bytes);
        tma_load_2d(sI + s * stage_words, &mapPl, &bars[s], I * kTile, ch * B);
        tma_load_2d(sJ + s * stage_words, &mapPl, &bars[s], J * kTile, ch * B);
    };

    // done[s]: warps finished with stage s's current chunk. The last of them refills the stage
    // (see the end of the chunk loop), so no warp waits for another except on the data.
    __shared__ uint32_t done[kBitStages];
    if (threadIdx.x < kBitStages) done[threadIdx.x] = 0u;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kBitStages; ++s) mbar_init(&bars[s], 1);
        fence_barrier_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int I, J, ch = chunks;
        for (int s = 0; s < kBitStages && s < units; ++s, ++ch) {
            if (ch == chunks) locate(s, I, J, ch);
            load(s, I, J, ch);
        }
    }
    // 16 warps: rows row0..row0+7 and columns col0..col0+3 of the tile per thread. A warp's 8
    // column groups read 128 contiguous bytes of a plane; its 4 row groups read 4 x 32 bytes.
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cb = warp >> 2, rb = ((warp & 3) + (cb == 1 || cb == 2 ? 3 : 0)) & 3;
    const int row0 = rb * 32 + (lane >> 3) * 8;
    const int col0 = cb * 32 + (lane & 7) * 4;

    const bool wide = ld_out % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    bool ok = true;
    int s = 0;           // the next unit's stage and its phase
    uint32_t phase = 0;
    int64_t n = 0;       // the tile's first unit
#pragma unroll 1
    while (n < units) {
        int I, J, ch0;
        locate(n, I, J, ch0);
        const int ch1 = int(units - n < chunks - ch0 ? ch0 + (units - n) : chunks);
        const bool counts = I != J || rb <= cb;
        uint32_t acc[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0u;
#pragma unroll 1
        for (int ch = ch0; ch < ch1; ++ch) {
            if (ok && !mbar_wait_bounded(&bars[s], phase, kMaxPolls)) ok = false;
            if (ok && counts) {
                const uint32_t* pI = sI + s * stage_words;
                const uint32_t* pJ = sJ + s * stage_words;
                uint32_t br[8][4];
#pragma unroll
                for (int r = 0; r < 8; ++r)
#pragma unroll
                    for (int q = 0; q < 4; ++q) br[r][q] = 0u;
#pragma unroll
                for (int k = 0; k < B; ++k) {
                    uint32_t a[8], b[4];
                    const uint4 a0 = *reinterpret_cast<const uint4*>(pI + k * kTile + row0);
                    const uint4 a1 = *reinterpret_cast<const uint4*>(pI + k * kTile + row0 + 4);
                    const uint4 b0 = *reinterpret_cast<const uint4*>(pJ + k * kTile + col0);
                    a[0] = a0.x, a[1] = a0.y, a[2] = a0.z, a[3] = a0.w, a[4] = a1.x, a[5] = a1.y, a[6] = a1.z, a[7] = a1.w;
                    b[0] = b0.x, b[1] = b0.y, b[2] = b0.z, b[3] = b0.w;
#pragma unroll
                    for (int r = 0; r < 8; ++r)
#pragma unroll
                        for (int q = 0; q < 4; ++q) br[r][q] = borrow_step(a[r], b[q], br[r][q]);
                }
#pragma unroll
                for (int r = 0; r < 8; ++r)
#pragma unroll
                    for (int q = 0; q < 4; ++q) acc[r][q] += __popc(br[r][q]);
            }
            // This warp is done reading stage s. The last warp to get here refills it with unit
            // kBitStages further on: its lane 0 has seen every other warp's count (and, through the warp
            // barrier and the block fence, their reads of the stage come before the copy). Waiters
            // on bars[s] acquire the reset of done[s] with the stage's next phase.
            __syncwarp();
            if (lane == 0) {
                __threadfence_block();
                if (atomicAdd(&done[s], 1u) == uint32_t(kThreads / 32 - 1)) {
                    done[s] = 0u;
                    int nI = I, nJ = J, nch = ch + kBitStages;
                    const int64_t next = n + (nch - ch0);
                    if (ok && next < units) {
                        if (nch >= ch1) locate(next, nI, nJ, nch);
                        fence_proxy_async();
                        load(s, nI, nJ, nch);
                    }
                }
            }
            if (++s == kBitStages) s = 0, phase ^= 1u;
        }
        n += ch1 - ch0;
        if (!ok) break;
        if (!counts) continue;
        // Voters with a permutation ballot: each of them is counted in exactly one of d[i][j] and
        // d[j][i]. Irregular ballots (place 0 everywhere) are in neither and are added apart.
        uint32_t irregular = 0u;
        for (int c = ch0 + lane; c < ch1; c += 32) irregular += irr_chunk[c];
#pragma unroll
        for (int o = 16; o; o >>= 1) irregular += __shfl_xor_sync(0xffffffffu, irregular, o);
        const int64_t vlo = int64_t(ch0) * kVC, vhi = int64_t(ch1) * kVC < V ? int64_t(ch1) * kVC : V;
        const uint32_t Vu = uint32_t(vhi - vlo) - irregular;
        const bool split = ch1 - ch0 < chunks;
        const bool mirror = I != J || rb != cb;
        // A whole tile inside the matrix: the thread's cells, in 16-byte groups where the rows are aligned, and
        // the mirror image of the warp's 32 x 32 block row by row, 128 contiguous bytes at a time, after
        // an exchange of the thread's 8 rows with the 8 threads that share them (stored as they lie, its
        // cells cost a sector each). What is added to is read in groups first. One B200, us, with
        // scalar stores of the mirror image and sums cell by cell / so: C = 10001, V = 1000 1946 / 1769,
        // accumulating 2107 / 1713; C = V = 4096 1044 / 1031, 1059 / 1017; C = 2048, V = 1500 accumulating
        // 155 / 140.
        if (!split && (J + 1) * kTile <= C) {
            const int64_t i0 = int64_t(I) * kTile + row0, j0 = int64_t(J) * kTile + col0;
            uint32_t* const ij = out + i0 * ld_out + j0;
#pragma unroll
            for (int h = 0; h < 8; h += 4) {
                uint32_t v[4][4];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    if (!accumulate) {
#pragma unroll
                        for (int q = 0; q < 4; ++q) v[r][q] = 0u;
                    } else if (wide) {
                        const uint4 x = *reinterpret_cast<const uint4*>(ij + (h + r) * ld_out);
                        v[r][0] = x.x, v[r][1] = x.y, v[r][2] = x.z, v[r][3] = x.w;
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; ++q) v[r][q] = ij[(h + r) * ld_out + q];
                    }
                }
#pragma unroll
                for (int r = 0; r < 4; ++r) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) v[r][q] += i0 + h + r == j0 + q ? 0u : acc[h + r][q];
                    if (wide) {
                        *reinterpret_cast<uint4*>(ij + (h + r) * ld_out) =
                            make_uint4(v[r][0], v[r][1], v[r][2], v[r][3]);
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; ++q) ij[(h + r) * ld_out + q] = v[r][q];
                    }
                }
            }
            if (!mirror) continue;
            uint32_t* const ji = out + (int64_t(J) * kTile + cb * 32) * ld_out + int64_t(I) * kTile + rb * 32 + lane;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                uint32_t m[8], was[8];
#pragma unroll
                for (int t = 0; t < 8; ++t) was[t] = accumulate ? ji[(4 * t + q) * ld_out] : 0u;
#pragma unroll
                for (int r = 0; r < 8; ++r) m[r] = Vu - acc[r][q];
#pragma unroll
                for (int d = 4; d >= 1; d >>= 1) {
#pragma unroll
                    for (int r = 0; r < 8; ++r) {
                        if (r & d) continue;
                        const uint32_t got = __shfl_xor_sync(0xFFFFFFFFu, lane & d ? m[r] : m[r + d], d);
                        if (lane & d) m[r] = got;
                        else m[r + d] = got;
                    }
                }
#pragma unroll
                for (int t = 0; t < 8; ++t) ji[(4 * t + q) * ld_out] = was[t] + m[t];
            }
            continue;
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int i = I * kTile + row0 + r;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int j = J * kTile + col0 + q;
                const uint32_t c = acc[r][q];
                if (i < C && j < C) {
                    uint32_t* ij = out + int64_t(i) * ld_out + j;
                    uint32_t* ji = out + int64_t(j) * ld_out + i;
                    if (split || accumulate) {
                        if (i != j) atomicAdd(ij, c);
                        if (mirror) atomicAdd(ji, Vu - c);
                    } else {
                        *ij = i == j ? 0u : c;
                        if (mirror) *ji = Vu - c;
                    }
                }
            }
        }
    }
    if (!ok) raise_device_error(err, kErrTimeout);
}

// The pairs of the irregular ballots, as the reference counts them (py:46-48 over the ballot
// completed by py:75-83): with r the ballot as given (length len, ids in [0, C)) and M the ids
// absent from it in ascending order, appended only when len != C, the completed ballot is
// r ++ M and every position a before position b adds one to d[x_a][x_b]:
//   1. a < b within r;
//   2. every a of r with every m of M;
//   3. m1 < m2 within M.
// Every warp of the grid takes rows (a, or m1) of one ballot at a time, its lanes stride the
// partners, and each adds with an atomic. Each CTA keeps the ballot's presence bitmap
// (ceil(C / 32) words of dynamic shared memory) for 2 and 3. A call without irregular
// ballots returns at once.
constexpr int kIrrThreads = 512;
constexpr int kIrrMaxSmem = (1 << 20) / 8;  // the bitmap at the largest C (2^20 candidates)

template <typename Id>
__global__ void __launch_bounds__(kIrrThreads)
    irregular_kernel(const Id* __restrict__ ids, const int64_t* __restrict__ offsets, int64_t id_base, int C,
                     const uint32_t* __restrict__ irr_n, const uint32_t* __restrict__ irr_list,
                     const uint32_t* __restrict__ err, uint32_t* __restrict__ out, int64_t ld_out) {
    extern __shared__ uint32_t present[];
    const uint32_t n = *irr_n;
    if (n == 0u || *err == kErrOffsets) return;
    const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int64_t gw = int64_t(blockIdx.x) * warps + (threadIdx.x >> 5);
    const int64_t GW = int64_t(gridDim.x) * warps;
    const int words = (C + 31) >> 5;
    for (uint32_t q = 0; q < n; ++q) {
        const int64_t v = irr_list[q];
        const int64_t beg = offsets ? offsets[v] - id_base : v * C;
        const int64_t len = offsets ? offsets[v + 1] - offsets[v] : C;
        const Id* r = ids + beg;
        for (int64_t a = gw; a < len; a += GW) {
            uint32_t* row = out + int64_t(r[a]) * ld_out;
            for (int64_t b = a + 1 + lane; b < len; b += 32) atomicAdd(row + int64_t(r[b]), 1u);
        }
        if (len == int64_t(C)) continue;  // the same for every thread of the block
        __syncthreads();                  // the previous ballot's bitmap is no longer read
        for (int w = threadIdx.x; w < words; w += blockDim.x) present[w] = 0u;
        __syncthreads();
        for (int64_t a = threadIdx.x; a < len; a += blockDim.x) {
            const uint32_t id = uint32_t(r[a]);
            atomicOr(present + (id >> 5), 1u << (id & 31));
        }
        __syncthreads();
        auto absent = [&](int c) { return !((present[c >> 5] >> (c & 31)) & 1u); };
        for (int64_t a = gw; a < len; a += GW) {
            uint32_t* row = out + int64_t(r[a]) * ld_out;
            for (int m = lane; m < C; m += 32)
                if (absent(m)) atomicAdd(row + m, 1u);
        }
        for (int64_t m1 = gw; m1 < C; m1 += GW) {
            if (!absent(int(m1))) continue;
            uint32_t* row = out + m1 * ld_out;
            for (int64_t m2 = m1 + 1 + lane; m2 < C; m2 += 32)
                if (absent(int(m2))) atomicAdd(row + m2, 1u);
        }
    }
}

// The pack and count kernels for each plane count 1 .. kMaxPlanes.
template <typename Id>
using FusedKernel = void (*)(const Id*, const int64_t*, int64_t, int64_t, int, int, uint32_t*, Irregular, int64_t,
                             uint32_t*);

struct TallyKernels {
    void (*pack)(const float*, int64_t, int64_t, uint32_t*);
    void (*count)(CUtensorMap, int64_t, int, int, CountSplit, uint32_t*, int64_t, bool, const uint32_t*, uint32_t*);
    FusedKernel<uint8_t> fused8;  // places + planes for C < 2048 (B <= 11), else null
    FusedKernel<uint16_t> fused16;
    FusedKernel<int32_t> fused32;
};

template <int B> constexpr TallyKernels tally_entry() {
    if constexpr (B <= 11)
        return {pack_planes_kernel<B>, count_bits_kernel<B>, places_planes_kernel<uint8_t, B>,
                places_planes_kernel<uint16_t, B>, places_planes_kernel<int32_t, B>};
    else
        return {pack_planes_kernel<B>, count_bits_kernel<B>, nullptr, nullptr, nullptr};
}

template <int... Bs> struct TallyTable {
    static const TallyKernels* get() {
        static const TallyKernels t[] = {{nullptr, nullptr, nullptr, nullptr, nullptr}, tally_entry<Bs>()...};
        return t;
    }
};

const TallyKernels& tally_kernels(int B) {
    return TallyTable<1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 18, 19, 20>::get()[B];
}
static_assert(kMaxPlanes == 20, "the table instantiates planes 1 .. 20");

}  // namespace tally
}  // namespace se

using namespace se;
using namespace se::tally;

// Error word (256 B); the irregular-ballot record (16 B header holding the count, then one
// word per 32-voter chunk, then the ballot list, V words); the places f32 [V][Cq] (only from
// C = 2048 on: below that the places stay in shared memory); the bit planes u32
// [ceil(V/32) * B][Cq].
static int64_t chunks_of(int64_t V) { return (std::max<int64_t>(V, 1) + kVC - 1) / kVC; }
static int64_t irregular_header_bytes(int64_t V) { return 16 + 4 * chunks_of(V); }
static int64_t places_offset(int64_t V) {
    return 256 + round_up(irregular_header_bytes(V) + 4 * std::max<int64_t>(V, 1), 256);
}
static int64_t planes_offset(int64_t V, int C) {
    return C < kFusedMaxCq ? places_offset(V) : places_offset(V) + round_up(std::max<int64_t>(V, 1) * padded(C) * 4, 256);
}

extern "C" int64_t se_tally_workspace_bytes(int64_t V, int C) {
    if (V < 0 || C < 1) return -1;
    return planes_offset(V, C) + round_up(chunks_of(V) * planes_for(C) * padded(C) * 4, 256);
}

namespace {
se_status_t tally_impl(const void* d_ids, int id_bytes, const int64_t* d_offsets, int64_t id_base, int64_t V, int C,
                       unsigned flags, uint32_t* d_out, int64_t ld_out, void* d_work, int64_t work_bytes,
                       void* stream_, int64_t num_ids = -1) {
    clear_error();
    SE_REQUIRE(C >= 1 && C <= (1 << 20), SE_ERR_INVALID, "Number of candidates out of range (%d)", C);
    SE_REQUIRE(V >= 0 && V < (int64_t(1) << 24), SE_ERR_INVALID, "Number of voters out of range (%lld)",
               (long long)V);
    SE_REQUIRE(d_out != nullptr && ld_out >= C, SE_ERR_INVALID, "bad output matrix");
    SE_REQUIRE(id_bytes == 1 || id_bytes == 2 || id_bytes == 4, SE_ERR_INVALID, "id width must be 1, 2 or 4 bytes");
    SE_REQUIRE((flags & ~unsigned(SE_TALLY_ACCUMULATE | SE_TALLY_NO_SYNC | SE_TALLY_KEEP_ERROR)) == 0,
               SE_ERR_INVALID, "unknown tally flags %u", flags);
    SE_REQUIRE(V == 0 || d_ids, SE_ERR_INVALID, "null ballot pointer");
    SE_REQUIRE(d_offsets == nullptr || id_base >= 0, SE_ERR_INVALID, "negative id base");
    SE_REQUIRE((reinterpret_cast<uintptr_t>(d_ids) % unsigned(id_bytes)) == 0, SE_ERR_INVALID,
               "ballot ids are not aligned to their width");
    const bool accumulate = flags & SE_TALLY_ACCUMULATE;
    const bool check = !(flags & SE_TALLY_NO_SYNC);
    const int64_t need = se_tally_workspace_bytes(V, C);
    SE_REQUIRE(d_work != nullptr && work_bytes >= need, SE_ERR_WORKSPACE,
               "workspace of %lld bytes is smaller than the %lld bytes required", (long long)work_bytes,
               (long long)need);
    SE_REQUIRE((reinterpret_cast<uintptr_t>(d_work) & 255) == 0, SE_ERR_INVALID, "workspace must be 256-byte aligned");
    cudaStream_t s = static_cast<cudaStream_t>(stream_);
    uint8_t* work = static_cast<uint8_t*>(d_work);
    uint32_t* err = reinterpret_cast<uint32_t*>(work);
    Irregular irr;
    irr.n = reinterpret_cast<uint32_t*>(work + 256);
    irr.chunk = irr.n + 4;
    irr.list = irr.chunk + chunks_of(V);
    float* pos = reinterpret_cast<float*>(work + places_offset(V));
    const int64_t Cq = padded(C);
    const int R = int(Cq / kTile);

    if (!(flags & SE_TALLY_KEEP_ERROR)) SE_CUDA_TRY(cudaMemsetAsync(work, 0, 256, s));
    if (V == 0) {
        if (!accumulate) SE_CUDA_TRY(cudaMemset2DAsync(d_out, size_t(ld_out) * 4, 0, size_t(C) * 4, size_t(C), s));
        return SE_OK;
    }
    SE_CUDA_TRY(cudaMemsetAsync(irr.n, 0, size_t(irregular_header_bytes(V)), s));
    const int B = planes_for(C);
    const TallyKernels& K = tally_kernels(B);
    if (se_status_t st = raise_smem_limit(reinterpret_cast<const void*>(K.count), int(bits_smem(B)), "the tally kernel"))
        return st;
    const int64_t nch_all = (V + kVC - 1) / kVC;
    uint32_t* planes = reinterpret_cast<uint32_t*>(work + planes_offset(V, C));
    if (C < kFusedMaxCq) {  // places and planes in one pass, places in shared memory
        const size_t smem = fused_smem(Cq);
        const int w = id_bytes == 1 ? 0 : id_bytes == 2 ? 1 : 2;
        const void* fn = w == 0 ? reinterpret_cast<const void*>(K.fused8)
                       : w == 1 ? reinterpret_cast<const void*>(K.fused16)
                                : reinterpret_cast<const void*>(K.fused32);
        if (se_status_t st = raise_smem_limit(fn, int(fused_smem(kFusedMaxCq)), "the places kernel")) return st;
        if (w == 0)
            K.fused8<<<unsigned(nch_all), 1024, smem, s>>>(static_cast<const uint8_t*>(d_ids), d_offsets, id_base, V, C,
                                                           int(Cq), planes, irr, num_ids, err);
        else if (w == 1)
            K.fused16<<<unsigned(nch_all), 1024, smem, s>>>(static_cast<const uint16_t*>(d_ids), d_offsets, id_base, V,
                                                            C, int(Cq), planes, irr, num_ids, err);
        else
            K.fused32<<<unsigned(nch_all), 1024, smem, s>>>(static_cast<const int32_t*>(d_ids), d_offsets, id_base, V,
                                                            C, int(Cq), planes, irr, num_ids, err);
        SE_CHECK_LAUNCH();
    } else {
        if (id_bytes == 4)
            launch_positions(static_cast<const int32_t*>(d_ids), d_offsets, id_base, V, C, Cq, pos, irr, num_ids, err,
                             s);
        else if (id_bytes == 2)
            launch_positions(static_cast<const uint16_t*>(d_ids), d_offsets, id_base, V, C, Cq, pos, irr, num_ids, err,
                             s);
        else
            launch_positions(static_cast<const uint8_t*>(d_ids), d_offsets, id_base, V, C, Cq, pos, irr, num_ids, err,
                             s);
        SE_CHECK_LAUNCH();
        K.pack<<<dim3(unsigned(nch_all), unsigned((Cq + 255) / 256)), 256, 0, s>>>(pos, V, Cq, planes);
        SE_CHECK_LAUNCH();
    }
    CUtensorMap map;
    if (se_status_t st = se::closure::make_map(&map, planes, uint64_t(Cq), uint64_t(nch_all * B), uint64_t(Cq) * 4,
                                               kTile, uint32_t(B)))
        return st;
    // One CTA per SM (fewer when there are not two 32-voter chunks for each), all whole tiles that
    // come out even, then the rest of the tiles cut into equal ranges (CountSplit). Cutting pays
    // when the wait for the last whole tiles is longer than what it adds: an output by atomic adds
    // at each end of a range and the zeroing before it. Costs in microseconds, measured on B200:
    // counting 0.15 per 32-voter chunk and plane-plus-two, a whole tile's output 3, cutting 27 where
    // counts are added to out and 39 where it is zeroed first. Whole / cut, us: C = 2048, V = 3000
    // 235 / 256, 5000 365 / 378, 7000 496 / 490, adding 238 / 248, 365 / 364, 494 / 481; C = 1900, V =
    // 700 99 / 119, 2500 201 / 204, adding 101 / 111, 201 / 196; C = 4000, V = 500 191 / 207, 1500 451 / 436;
    // C = 8000, V = 800 861 / 865, adding 862 / 857; C = 1000, V = 1500 128 / 104.
    int sms = 0, dev = 0;
    SE_CUDA_TRY(cudaGetDevice(&dev));
    SE_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int64_t chunks = (V + kVC - 1) / kVC;
    const int64_t tiles = int64_t(R) * (R + 1) / 2;
    const int64_t grid = std::min<int64_t>(sms, std::max<int64_t>(tiles, tiles * chunks / 2));
    const double full_us = 0.15 * double(chunks) * double(B + 2);
    CountSplit layout{tiles_above(R) / grid, false};
    const int64_t above = tiles_above(R) - layout.rounds * grid;
    const double cut_us = (double(above) + 0.8 * R) / double(grid) * full_us + (accumulate ? 27.0 : 39.0);
    layout.whole = double((above + R + grid - 1) / grid) * (full_us + 3.0) <= cut_us;
    if (!accumulate && !layout.whole && grid > 1) {
        zero_tiles_kernel<<<dim3(unsigned(grid - 1), kZeroParts), 256, 0, s>>>(d_out, ld_out, C, R, chunks, layout, err);
        SE_CHECK_LAUNCH();
    }
    K.count<<<unsigned(grid), kThreads, bits_smem(B), s>>>(map, V, C, R, layout, d_out, ld_out, accumulate, irr.chunk,
                                                           err);
    SE_CHECK_LAUNCH();
    // The irregular ballots' pairs, after the count's stores. Without any it returns at once.
    const size_t irr_smem = size_t((C + 31) / 32) * 4;
    const unsigned irr_grid = unsigned(2 * sms);
    if (id_bytes == 4) {
        auto fn = irregular_kernel<int32_t>;
        if (se_status_t st = raise_smem_limit(reinterpret_cast<const void*>(fn), kIrrMaxSmem, "the irregular-ballot kernel"))
            return st;
        fn<<<irr_grid, kIrrThreads, irr_smem, s>>>(static_cast<const int32_t*>(d_ids), d_offsets, id_base, C, irr.n,
                                                  irr.list, err, d_out, ld_out);
    } else if (id_bytes == 2) {
        auto fn = irregular_kernel<uint16_t>;
        if (se_status_t st = raise_smem_limit(reinterpret_cast<const void*>(fn), kIrrMaxSmem, "the irregular-ballot kernel"))
            return st;
        fn<<<irr_grid, kIrrThreads, irr_smem, s>>>(static_cast<const uint16_t*>(d_ids), d_offsets, id_base, C, irr.n,
                                                  irr.list, err, d_out, ld_out);
    } else {
        auto fn = irregular_kernel<uint8_t>;
        if (se_status_t st = raise_smem_limit(reinterpret_cast<const void*>(fn), kIrrMaxSmem, "the irregular-ballot kernel"))
            return st;
        fn<<<irr_grid, kIrrThreads, irr_smem, s>>>(static_cast<const uint8_t*>(d_ids), d_offsets, id_base, C, irr.n,
                                                  irr.list, err, d_out, ld_out);
    }
    SE_CHECK_LAUNCH();
    if (!check) return SE_OK;

    uint32_t code = 0;
    SE_CUDA_TRY(cudaMemcpyAsync(&code, err, 4, cudaMemcpyDeviceToHost, s));
    SE_CUDA_TRY(cudaStreamSynchronize(s));
    SE_REQUIRE(code != kErrOffsets, SE_ERR_INVALID, "offsets must start at 0, never decrease and end at len(ids)");
    SE_REQUIRE(code != kErrRange, SE_ERR_DEVICE, "a ballot names a candidate outside [0, %d)", C);
    SE_REQUIRE(code == 0, SE_ERR_DEVICE, "tally kernel reported device error %u (TMA wait timed out)", code);
    return SE_OK;
}
}  // namespace

extern "C" se_status_t se_tally(const int32_t* d_ids, const int64_t* d_offsets, int64_t V, int C, uint32_t* d_out,
                                int64_t ld_out, void* d_work, int64_t work_bytes, void* stream) {
    clear_error();
    SE_REQUIRE(V == 0 || d_offsets != nullptr, SE_ERR_INVALID, "null ballot pointer");
    return tally_impl(d_ids, 4, d_offsets, 0, V, C, 0u, d_out, ld_out, d_work, work_bytes, stream);
}

extern "C" se_status_t se_tally_checked(const int32_t* d_ids, int64_t num_ids, const int64_t* d_offsets, int64_t V,
                                        int C, uint32_t* d_out, int64_t ld_out, void* d_work, int64_t work_bytes,
                                        void* stream) {
    clear_error();
    SE_REQUIRE(V == 0 || d_offsets != nullptr, SE_ERR_INVALID, "null ballot pointer");
    SE_REQUIRE(num_ids >= 0, SE_ERR_INVALID, "negative number of ids");
    return tally_impl(d_ids, 4, d_offsets, 0, V, C, 0u, d_out, ld_out, d_work, work_bytes, stream, num_ids);
}

extern "C" se_status_t se_tally_enqueue(const int32_t* d_ids, const int64_t* d_offsets, int64_t V, int C,
                                        uint32_t* d_out, int64_t ld_out, void* d_work, int64_t work_bytes,
                                        void* stream) {
    clear_error();
    SE_REQUIRE(V == 0 || d_offsets != nullptr, SE_ERR_INVALID, "null ballot pointer");
    return tally_impl(d_ids, 4, d_offsets, 0, V, C, SE_TALLY_NO_SYNC, d_out, ld_out, d_work, work_bytes, stream);
}

extern "C" se_status_t se_tally_ex(const void* d_ids, int id_bytes, const int64_t* d_offsets, int64_t id_base,
                                   int64_t V, int C, unsigned flags, uint32_t* d_out, int64_t ld_out, void* d_work,
                                   int64_t work_bytes, void* stream) {
    return tally_impl(d_ids, id_bytes, d_offsets, id_base, V, C, flags, d_out, ld_out, d_work, work_bytes, stream);
}
