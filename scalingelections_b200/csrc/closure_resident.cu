// One-launch closure of a small matrix: the whole working matrix stays in registers.
//
// Up to C = 1536 (16-bit lanes) the padded matrix fits the register files of the GPU's SMs with room. The
// schedules of closure.cu keep it in L2 and run two launches per 128-pivot round; at these sizes
// their time is the serial chain of a round (close the 128-pivot tile, the panels, the next
// diagonal tile, two launches), about 52 us a round whatever the size, with most SMs idle. Here
//   * one cooperative launch runs the defeat init, every round and the widened output;
//   * each CTA (one or two per SM) owns a row of CB blocks of 64 x 64 cells and keeps them in registers;
//   * a round has 32 pivots, half a block: what is serial in a round (closing a 32 x 32 piece, its
//     product with the next row and column pieces, the next diagonal piece) is short;
//   * there is no barrier between rounds. Round k's panel blocks A[k][i] (its pivot columns in
//     block row i, transposed) and B[k][j] (its pivot rows in block column j) are published to
//     global memory, each with a flag, and a CTA waits only for the blocks of its own row and
//     columns. Every round has panel buffers of its own, so nothing published is overwritten.
//
// Round k, with K its pivots, D the 32 x 32 diagonal piece S[K][K] and (x) the max-min product:
//   D       closed, by two warps of the CTA that owns it;
//   S[K][j] = max(S[K][j], D (x) S[K][j])   by the owners of those rows;     published as B[k][j]
//   S[i][K] = max(S[i][K], S[i][K] (x) D)   by the owners of those columns;  published as A[k][i]
//   S[i][j] = max(S[i][j], A[k][i] (x) B[k][j])  everywhere else.
// An owner of round k + 1's rows or columns takes those pieces of round k first, then does its part
// of round k + 1's diagonal or panels, and only then the rest of round k, so that the chain runs
// ahead of the bulk. A cell may meet a round's product a second time there: every product is a
// path's strength, so a repeated one changes nothing.
//
// A block's two rounds (k even, k + 1) follow each other in the CTA that owns the diagonal block,
// whose four 32 x 32 pieces belong to four pairs of warps (diagonal()). What the chain needs from
// another CTA goes through mailboxes whose 8-byte packets hold a word and a tag: D of both rounds,
// the two other pieces of the diagonal block in round k (with which the panels' owners bring their
// round k + 1 cells up to date) and the pieces of round k + 1's panels that the next diagonal block
// is updated with. The receiver polls the data itself: about 0.7 us from CTA to CTA, against 2.5 us
// for data, fence, flag and copy.
//
// Inside a CTA the warps run apart: a panel takes the four warps that hold its half of a block,
// while the others go on with the bulk, and a slot of shared memory is handed from its writers
// to its readers, and back, through mbarriers. Helper warps: the producer watches the flags and
// brings each published block into its slot as one bulk copy (blocks are stored exactly as the
// product reads them); two publishers, for the row and the columns, raise the flags of the CTA's
// own blocks, so that no compute warp waits for a fence.
//
// All CTAs of the launch have to be on the GPU at once, and kernels of other streams may hold SMs for
// as long as they like. So the CTAs check in before the first round (all_here): if they are not all
// there within a limit, the launch gives way, that is, every CTA leaves before anything is
// written but flags, and the closure runs as launches, which take the room there is: started by
// the host where the call waits, or by kernels queued behind this one that otherwise return at
// once (closure.cu). A checked-in launch has its SMs until it ends.
//
// Every wait is bounded. A wait that runs out records an error and makes its thread stop waiting,
// not stop: control flow stays uniform, every CTA reaches the end, and the host reports the error. A
// thread that has given up arrives on no barrier of the slots any more, so nobody who still waits is
// told that a slot is full or free when it is not, and no barrier gets more arrivals than it counts. The
// producer that gives up starts no more copies and waits for those that it started.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>

#include "closure_core.cuh"
#include "closure_resident.cuh"

namespace se {
namespace resident {

using closure::cell_splat;
using closure::kErrTmaTimeout;
using closure::ld4;
using closure::st4;

constexpr uint64_t kWaitNs = 2000000000ull;  // one wait, unless the caller sets another limit
constexpr int kP = 32;               // pivots per round
constexpr int kNT = 256;             // compute threads
constexpr int kThreads = kNT + 96;  // and the helper warps: the producer and two publishers

// Words of the flags area at the start of the workspace. 0 and 1 are the closure's common words
// (device error, 16-bit overflow).
constexpr int kWordErr = 0, kWordOverflow = 1, kWordLo = 2, kWordHi = 3, kWordWide = kWide, kWordArrived = kArrived;

// Thread geometry: the compute threads share every 64 x 64 block evenly, 4 x 4 cells each: thread
// (tr, tc) owns rows 4 tr .. and cells 4 tc .. of each of the CTA's blocks. A warp is 4 x 8 threads:
// 16 rows (group rg) of one column half. Warps 4..7 take the halves in the other order, so that
// the four warps of a row half, and those of a column half, run on different schedulers.
template <int LB> struct geo {
    static constexpr int CPW = 32 / LB;
    static constexpr int WPB = kB / CPW;     // words per block row
    static constexpr int QR = 4;             // rows
    static constexpr int QC = 4 / CPW;       // and words per thread and block
    static constexpr int QW = QR * QC;
    static constexpr int A_WORDS = kP * kB;  // one A block (u16 cells duplicated into both halves)
    static constexpr int B_WORDS = kP * WPB; // one B block
    static constexpr int PA_WORDS = kP * kP;         // a 32 x 32 piece in A form
    static constexpr int PB_WORDS = kP * (WPB / 2);  // and in B form
    // A block's mailboxes, in packets: D of its two rounds, the sides of its diagonal block in the
    // first (A form, B form), and of each round the panels' pieces for the next diagonal block.
    static constexpr int MAIL_D = 0, MAIL_SIDE_A = 128 * QW, MAIL_SIDE_B = 192 * QW, MAIL_A = 256 * QW,
                         MAIL_B = 512 * QW, MAIL = 768 * QW;
};

// N consecutive words, N = 1, 2 or 4, naturally aligned.
template <int N> __device__ __forceinline__ void ldn(uint32_t* dst, const uint32_t* src) {
    if constexpr (N == 4) {
        ld4(dst, src);
    } else {
        const uint2 v = *reinterpret_cast<const uint2*>(src);
        dst[0] = v.x, dst[1] = v.y;
    }
}
template <int N> __device__ __forceinline__ void stn(uint32_t* dst, const uint32_t* src) {
    if constexpr (N == 4) st4(dst, src);
    else *reinterpret_cast<uint2*>(dst) = make_uint2(src[0], src[1]);
}

__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_gpu(uint32_t* p, uint32_t v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire_smem(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_smem(uint32_t* p, uint32_t v) {
    asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

// One contiguous block of global memory into shared memory; both 16-byte aligned.
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(smem_dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// Named barriers. Warps pair up by the 32 x 32 piece of each block that they hold (rows of half rh,
// cells of half ch); four warps share a row half, and four a column half. Not the .aligned forms:
// these follow branches on the lane.
template <int N> __device__ __forceinline__ void sync_threads(int id) {
    __syncwarp();
    asm volatile("barrier.sync %0, %1;" ::"r"(id), "n"(N) : "memory");
}
template <int N> __device__ __forceinline__ void arrive_threads(int id) {
    __syncwarp();
    asm volatile("barrier.arrive %0, %1;" ::"r"(id), "n"(N) : "memory");
}
__device__ __forceinline__ void sync_compute() { sync_threads<kNT>(1); }
__device__ __forceinline__ void sync_pair(int pair) { sync_threads<64>(2 + pair); }
__device__ __forceinline__ void sync_rows(int h) { sync_threads<128>(6 + h); }
__device__ __forceinline__ void sync_cols(int h) { sync_threads<128>(8 + h); }
constexpr int kBarD = 10, kBarSides = 11;  // the diagonal block's D is there; its other two pieces are
constexpr int kBarEnd = 12;                // the compute warps are done with the slots

struct Params {
    const uint32_t* d;
    int64_t ld;
    uint32_t* out;
    int64_t ld_out;
    uint32_t* words;   // flags area (kWord*)
    uint32_t* flag_a;  // [NR][NB]: A[k][i] published
    uint32_t* flag_b;  // [NR][NB]: B[k][j] published
    uint64_t* mail;    // [NB] blocks' mailboxes (MAIL_* in geo)
    uint32_t* A;       // [NR][NB] blocks
    uint32_t* B;       // [NR][NB] blocks
    int C, NB, NR, tiles_j;
    uint32_t base;     // 16-bit lanes store a kept value v as v - base (see init_kernel in closure.cu)
    int automatic;     // choose the 16-bit window here; give up (kWordWide) when none holds
    uint64_t start_ns; // the check-in's limit
    uint64_t wait_ns;  // the limit of any wait after it; 0: one look
    uint32_t polls;    // and that of a wait on an mbarrier
};

// One thread of each CTA checks in and waits for the others. All of them see the same outcome: a wait
// that runs out can mark the word only as long as a CTA is missing from its count, and a marked
// count never serves as a full one.
__device__ __forceinline__ bool all_here(uint32_t* arrived, uint32_t n, uint64_t limit_ns) {
    if (limit_ns == 0u && n > 1u) {  // no wait at all, for every CTA alike
        atomicOr(arrived, kGaveWay);
        return false;
    }
    __threadfence();
    uint32_t seen = atomicAdd(arrived, 1u) + 1u;
    const uint64_t t0 = global_ns();
    for (uint32_t it = 0; seen != n && !(seen & kGaveWay); ++it) {
        if ((it & 63u) == 0u && global_ns() - t0 >= limit_ns) {
            const uint32_t old = atomicCAS(arrived, seen, seen | kGaveWay);
            seen = old == seen ? seen | kGaveWay : old;
        } else {
            seen = ld_acquire_gpu(arrived);
        }
    }
    __threadfence();
    return seen == n;
}

// c[r][q] = max(c[r][q], max_k min(A[k][row], B[k][word])) over kn pivots (a multiple of 4). a and
// b point at the thread's row and word; PA and PB are the operands' pitches.
template <int LB, int PA, int PB>
__device__ __forceinline__ void relax_block(uint32_t (&c)[geo<LB>::QR][geo<LB>::QC], const uint32_t* __restrict__ a,
                                            const uint32_t* __restrict__ b, int kn) {
    using G = geo<LB>;
    using L = lanes<LB>;
#pragma unroll 4
    for (int k = 0; k < kn; k += 2) {
        uint32_t a0[G::QR], a1[G::QR], b0[G::QC], b1[G::QC];
        ldn<G::QR>(a0, a + k * PA);
        ldn<G::QR>(a1, a + (k + 1) * PA);
        ldn<G::QC>(b0, b + k * PB);
        ldn<G::QC>(b1, b + (k + 1) * PB);
#pragma unroll
        for (int r = 0; r < G::QR; ++r)
#pragma unroll
            for (int q = 0; q < G::QC; ++q)
                c[r][q] = L::vmax3(c[r][q], L::vmin(a0[r], b0[q]), L::vmin(a1[r], b1[q]));
    }
}

// The same over N blocks side by side (consecutive B blocks); the A operand is read once.
template <int LB, int N, int PA, int PB>
__device__ __forceinline__ void relax_row(uint32_t (&c)[N][geo<LB>::QR][geo<LB>::QC], const uint32_t* __restrict__ a,
                                          const uint32_t* __restrict__ b, int kn) {
    using G = geo<LB>;
    using L = lanes<LB>;
#pragma unroll 2
    for (int k = 0; k < kn; k += 2) {
        uint32_t a0[G::QR], a1[G::QR];
        ldn<G::QR>(a0, a + k * PA);
        ldn<G::QR>(a1, a + (k + 1) * PA);
#pragma unroll
        for (int y = 0; y < N; ++y) {
            uint32_t b0[G::QC], b1[G::QC];
            ldn<G::QC>(b0, b + y * G::B_WORDS + k * PB);
            ldn<G::QC>(b1, b + y * G::B_WORDS + (k + 1) * PB);
#pragma unroll
            for (int r = 0; r < G::QR; ++r)
#pragma unroll
                for (int q = 0; q < G::QC; ++q)
                    c[y][r][q] = L::vmax3(c[y][r][q], L::vmin(a0[r], b0[q]), L::vmin(a1[r], b1[q]));
        }
    }
}
// A thread's cells as rows (B form: at points to its first row's words, PB the pitch) and transposed
// (A form: u16 cells duplicated; at points to its first cell's column, PA the pitch).
template <int LB, int PB>
__device__ __forceinline__ void store_b(const uint32_t (&c)[geo<LB>::QR][geo<LB>::QC], uint32_t* at) {
#pragma unroll
    for (int r = 0; r < geo<LB>::QR; ++r) stn<geo<LB>::QC>(at + r * PB, c[r]);
}
template <int LB, int PA>
__device__ __forceinline__ void store_a(const uint32_t (&c)[geo<LB>::QR][geo<LB>::QC], uint32_t* at) {
    using G = geo<LB>;
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        uint32_t v[G::QR];
#pragma unroll
        for (int r = 0; r < G::QR; ++r) v[r] = cell_splat<LB>(c[r][n / G::CPW], n % G::CPW);
        st4(at + n * PA, v);
    }
}

// Closes the 32 x 32 piece spread over a pair of warps (thread (lr, lc) of 8 x 8 holds 4 x 4
// cells), two pivots per barrier, by the scheme of close_tile_in_registers (closure_core.cuh): rows
// and columns k and k + 1 are published together and each thread applies step k to the row and
// column k + 1 that it reads. Pivots go in groups of 4, so the registers that hold a published row
// or column are indexed statically. kn: a multiple of 4.
template <int LB> struct ChainBuf {
    uint32_t row[4][geo<LB>::WPB / 2];
    uint32_t col[4][kP];
};

template <int LB, int J>
__device__ __forceinline__ void publish_pivot(const uint32_t (&c)[geo<LB>::QR][geo<LB>::QC], int lr, int lc, int g,
                                              uint32_t* row, uint32_t* col) {
    using G = geo<LB>;
    if (lr == g) stn<G::QC>(row + G::QC * lc, c[J]);
    if (lc == g) {
        uint32_t v[G::QR];
#pragma unroll
        for (int r = 0; r < G::QR; ++r) v[r] = cell_splat<LB>(c[r][J / G::CPW], J % G::CPW);
        st4(col + G::QR * lr, v);
    }
}

template <int LB, int J>
__device__ __forceinline__ void close_pair(uint32_t (&c)[geo<LB>::QR][geo<LB>::QC], int lr, int lc, int g,
                                           ChainBuf<LB>& buf, int pair) {
    using G = geo<LB>;
    using L = lanes<LB>;
    constexpr int s = J, t = J ^ 2;  // staging slots of this pair and of the next
    uint32_t a0[G::QR], a1[G::QR], b0[G::QC], b1[G::QC];
    ldn<G::QR>(a0, &buf.col[s][G::QR * lr]);
    ldn<G::QR>(a1, &buf.col[s + 1][G::QR * lr]);
    ldn<G::QC>(b0, &buf.row[s][G::QC * lc]);
    ldn<G::QC>(b1, &buf.row[s + 1][G::QC * lc]);
    const uint32_t ckk1 = cell_splat<LB>(buf.row[s][(4 * g + J + 1) / G::CPW], (J + 1) % G::CPW);  // c[k][k+1]
    const uint32_t ck1k = buf.col[s][4 * g + J + 1];                                             // c[k+1][k]
#pragma unroll
    for (int r = 0; r < G::QR; ++r) a1[r] = L::vmax(a1[r], L::vmin(a0[r], ckk1));
#pragma unroll
    for (int q = 0; q < G::QC; ++q) b1[q] = L::vmax(b1[q], L::vmin(ck1k, b0[q]));
#pragma unroll
    for (int r = 0; r < G::QR; ++r)
#pragma unroll
        for (int q = 0; q < G::QC; ++q) c[r][q] = L::vmax3(c[r][q], L::vmin(a0[r], b0[q]), L::vmin(a1[r], b1[q]));
    if constexpr (J == 0) {
        publish_pivot<LB, 2>(c, lr, lc, g, buf.row[t], buf.col[t]);
        publish_pivot<LB, 3>(c, lr, lc, g, buf.row[t + 1], buf.col[t + 1]);
    } else {  // past the last group no thread matches
        publish_pivot<LB, 0>(c, lr, lc, g + 1, buf.row[t], buf.col[t]);
        publish_pivot<LB, 1>(c, lr, lc, g + 1, buf.row[t + 1], buf.col[t + 1]);
    }
    sync_pair(pair);
}

template <int LB>
__device__ __forceinline__ void close_piece(uint32_t (&c)[geo<LB>::QR][geo<LB>::QC], int lr, int lc, int kn,
                                            ChainBuf<LB>& buf, int pair) {
    publish_pivot<LB, 0>(c, lr, lc, 0, buf.row[0], buf.col[0]);
    publish_pivot<LB, 1>(c, lr, lc, 0, buf.row[1], buf.col[1]);
    sync_pair(pair);
#pragma unroll 1
    for (int g = 0; 4 * g < kn; ++g) {
        close_pair<LB, 0>(c, lr, lc, g, buf, pair);
        close_pair<LB, 2>(c, lr, lc, g, buf, pair);
    }
}

// A piece through a mailbox: 64 threads send their fragments, 64 threads of another CTA (lt: the
// thread's place among them) receive them. Each 8-byte packet is one word and a tag; the mailboxes
// start at zero.
template <int LB>
__device__ __forceinline__ void send_piece(const uint32_t (&c)[geo<LB>::QR][geo<LB>::QC], uint64_t* box, int lt) {
    using G = geo<LB>;
#pragma unroll
    for (int i = 0; i < G::QW / 2; ++i)
        asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(box + (i * 64 + lt) * 2),
                     "l"(uint64_t(c[2 * i / G::QC][2 * i % G::QC]) | (1ull << 32)),
                     "l"(uint64_t(c[2 * i / G::QC][2 * i % G::QC + 1]) | (1ull << 32))
                     : "memory");
}
// One poll of a box: whether the whole fragment is there.
template <int LB>
__device__ __forceinline__ bool poll_piece(uint32_t (&c)[geo<LB>::QR][geo<LB>::QC], const uint64_t* box, int lt) {
    using G = geo<LB>;
    uint64_t all = ~0ull;
#pragma unroll
    for (int i = 0; i < G::QW / 2; ++i) {
        uint64_t x, y;
        asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];"
                     : "=l"(x), "=l"(y)
                     : "l"(box + (i * 64 + lt) * 2)
                     : "memory");
        c[2 * i / G::QC][2 * i % G::QC] = uint32_t(x);
        c[2 * i / G::QC][2 * i % G::QC + 1] = uint32_t(y);
        all &= x & y;
    }
    return uint32_t(all >> 32) == 1u;
}

// Four consecutive cells of row r from column c0; cells past C read as 0.
__device__ __forceinline__ void load_cells(uint32_t (&v)[4], const uint32_t* d, int64_t ld, int C, int r, int c0,
                                           bool vec) {
    const uint32_t* p = d + int64_t(r) * ld + c0;
    if (vec && r < C && c0 + 4 <= C) {
        ld4(v, p);
    } else {
#pragma unroll
        for (int n = 0; n < 4; ++n) v[n] = r < C && c0 + n < C ? p[n] : 0u;
    }
}

// The thread's share of block (bi, bj) of the defeat matrix: a cell d[i][j] is kept when it
// exceeds d[j][i]. lo and hi follow the kept values; over rises on a value outside the window.
template <int LB>
__device__ __forceinline__ void load_defeats(uint32_t (&c)[geo<LB>::QR][geo<LB>::QC], const Params& P, uint32_t base,
                                             int bi, int bj, int tr, int tc, bool vec, uint32_t& lo, uint32_t& hi,
                                             bool& over) {
    using G = geo<LB>;
    const int i0 = bi * kB + 4 * tr, j0 = bj * kB + 4 * tc;
    uint32_t x[4][4], y[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) load_cells(x[r], P.d, P.ld, P.C, i0 + r, j0, vec);
#pragma unroll
    for (int n = 0; n < 4; ++n) load_cells(y[n], P.d, P.ld, P.C, j0 + n, i0, vec);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < G::QC; ++q) {
            uint32_t w = 0u;
#pragma unroll
            for (int h = 0; h < G::CPW; ++h) {
                const int n = q * G::CPW + h;
                uint32_t v = x[r][n] > y[n][r] ? x[r][n] : 0u;
                if (v != 0u) {
                    lo = v < lo ? v : lo;
                    hi = v > hi ? v : hi;
                    if constexpr (LB == 16) {
                        if (v <= base || v - base > 0xFFFFu) {
                            over = true;
                            v = 0xFFFFu;
                        } else {
                            v -= base;
                        }
                    }
                }
                w |= LB == 16 ? v << (16 * h) : v;
            }
            c[r][q] = w;
        }
}

// Dynamic shared memory: the stages' A and B slots, D of the last even and odd round in both forms,
// each pair's piece of the diagonal block's work in both forms, a received side piece in both forms,
// and the closing's staging rows.
template <int LB, int CB, int kStages> struct smem_layout {
    using G = geo<LB>;
    static constexpr int STAGE = G::A_WORDS + CB * G::B_WORDS;
    static constexpr int DT = kStages * STAGE;
    static constexpr int DB = DT + 2 * G::PA_WORDS;
    static constexpr int PAIR_A = DB + 2 * G::PB_WORDS;
    static constexpr int PAIR_B = PAIR_A + 4 * G::PA_WORDS;
    static constexpr int SIDE_A = PAIR_B + 4 * G::PB_WORDS;
    static constexpr int SIDE_B = SIDE_A + G::PA_WORDS;
    static constexpr int CHAIN = SIDE_B + G::PB_WORDS;
    static constexpr int WORDS = CHAIN + int(sizeof(ChainBuf<LB>) / 4);
    static constexpr int BYTES = WORDS * 4;
};

template <int LB, int CB, int OCC, int kStages>
__global__ void __launch_bounds__(kThreads, OCC) resident_kernel(const __grid_constant__ Params P) {
    using G = geo<LB>;
    using SL = smem_layout<LB, CB, kStages>;
    constexpr int QR = G::QR, QC = G::QC, WH = G::WPB / 2;
    constexpr bool kEarly = CB == 1;  // diagonal() runs two rounds ahead
    extern __shared__ __align__(1024) uint32_t smem[];
    __shared__ uint64_t full[kStages][1 + CB], empty[kStages];  // slot 0 is A, slot 1 + y is B[y]
    __shared__ uint32_t s_lo, s_hi, s_base, s_go, s_dead;
    __shared__ uint32_t prog_row[kNT / 32], prog_col[kNT / 32];  // panel blocks stored, per warp
    const int I = blockIdx.x / P.tiles_j, J = blockIdx.x % P.tiles_j;
    const int NB = P.NB, NR = P.NR;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) {
            for (int x = 0; x < 1 + CB; ++x) mbar_init(&full[s][x], 1);
            mbar_init(&empty[s], kNT / 32);
        }
        fence_barrier_init();
        s_lo = 0xFFFFFFFFu;
        s_hi = 0u;
        s_go = 1u;
        s_dead = 0u;
        s_base = P.base;
    }
    if (tid < kNT / 32) prog_row[tid] = prog_col[tid] = 0u;
    __syncthreads();

    auto pivots = [&](int k) {  // pivots of round k, rounded up to a group of 4 (zero padding past C)
        const int n = P.C - k * kP;
        return n >= kP ? kP : (n + 3) & ~3;
    };
    const int nc = min(CB, NB - J * CB);  // blocks that hold candidates
    auto slot_a = [&](int k) { return smem + (k % kStages) * SL::STAGE; };
    auto slot_b = [&](int k, int y) { return smem + (k % kStages) * SL::STAGE + G::A_WORDS + y * G::B_WORDS; };
    auto in_rows = [&](int k) { return k < NR && (k >> 1) == I; };       // round k's pivots are rows of this CTA
    auto in_cols = [&](int k) { return k < NR && (k >> 1) / CB == J; };  // or columns
    auto col_of = [&](int k) { return (k >> 1) - J * CB; };
    // The row panel block that is stored first: the one that the next diagonal block waits for.
    auto next_col = [&](int k) { return (k >> 1) + 1 - J * CB; };  // the next block's column here, if in [0, nc)
    auto first_col = [&](int k) { return next_col(k) >= 0 && next_col(k) < nc ? next_col(k) : 0; };
    auto block_a = [&](int k) { return P.A + (int64_t(k) * NB + I) * G::A_WORDS; };
    auto block_b = [&](int k, int y) { return P.B + (int64_t(k) * NB + J * CB + y) * G::B_WORDS; };

    // ---- Helper warps. ----
    if (warp >= kNT / 32) {
        if (!P.automatic && warp == kNT / 32 && lane == 0 && !all_here(P.words + kWordArrived, gridDim.x, P.start_ns))
            s_go = 0u;
        __syncthreads();  // every CTA is here and, with automatic lanes, the window is agreed on
        if (!s_go) return;
        const int role = warp - kNT / 32;
        if (role == 0) {
            // Producer: lane x watches slot x; lane 0 alone fills them (a bulk copy's operands are
            // warp-uniform, so one lane at a time may issue it).
            bool dead = false;              // a wait ran out (uniform, as all below)
            uint64_t copied = 0;            // 16 bits per stage: slots copied into, and the last copy's phase
            const uint32_t empty_blocks = ((1u << (1 + CB)) - 1u) & ~((1u << (1 + nc)) - 1u);
            for (int k = 0; k < NR && !dead; ++k) {
                const int s = k % kStages;
                // The compute warps fill the slots of the CTA's own panel blocks.
                uint32_t pending = (in_cols(k) ? 0u : 1u) | (in_rows(k) ? 0u : ((1u << nc) - 1u) << 1);
                if ((pending | empty_blocks) && k >= kStages)
                    dead = __any_sync(0xFFFFFFFFu,
                                      !mbar_wait_bounded(&empty[s], uint32_t(k / kStages - 1) & 1u, P.polls, P.wait_ns));
                if (dead) break;
                const uint32_t* flag = lane == 0 ? P.flag_a + k * NB + I : P.flag_b + k * NB + J * CB + lane - 1;
                uint32_t got = 0u;
                const uint64_t t0 = global_ns();
                for (uint32_t it = 1; pending; ++it) {
                    const uint32_t ready =
                        __ballot_sync(0xFFFFFFFFu, ((pending >> lane) & 1u) && ld_acquire_gpu(flag) != 0u);
                    if (ready) {
                        __syncwarp();
                        if (lane == 0) {
                            fence_proxy_async_all();  // the blocks were written through the generic proxy
                            for (int x = 0; x < 1 + CB; ++x)
                                if ((ready >> x) & 1u) {
                                    const uint32_t bytes = (x == 0 ? G::A_WORDS : G::B_WORDS) * 4;
                                    mbar_arrive_expect_tx(&full[s][x], bytes);
                                    bulk_load(x == 0 ? slot_a(k) : slot_b(k, x - 1),
                                              x == 0 ? block_a(k) : block_b(k, x - 1), bytes, &full[s][x]);
                                }
                        }
                        __syncwarp();
                        pending &= ~ready;
                        got |= ready;
                    } else if (P.wait_ns == 0u ||
                               ((it & 255u) == 0u && __any_sync(0xFFFFFFFFu, global_ns() - t0 > P.wait_ns))) {
                        dead = true;
                        break;
                    }
                }
                if (lane == 0 && !dead) {
                    for (int x = 0; x < 1 + CB; ++x)
                        if ((empty_blocks >> x) & 1u) mbar_arrive(&full[s][x]);  // a phase without a copy
                }
                __syncwarp();
                const uint32_t odd = (k / kStages) & 1 ? got : 0u;
                copied = (copied & ~(uint64_t(got << 8) << (16 * s))) | (uint64_t(got | odd << 8) << (16 * s));
            }
            if (dead && lane == 0) {
                s_dead = 1u;
                raise_device_error(P.words + kWordErr, kErrTmaTimeout);
            }
            // No copy outlives the CTA. The compute warps have waited for every slot of every round, unless one
            // gave up: then the last copy into each slot is waited for here. (Where the compute warps filled
            // that slot again it has landed, but its phase cannot be told from the next one, and the short
            // limit runs out.)
            sync_threads<kNT + 32>(kBarEnd);
            if (lane == 0 && s_dead) {
                for (int s = 0; s < kStages; ++s)
                    for (int x = 0; x < 1 + CB; ++x) {
                        const uint32_t c = uint32_t(copied >> (16 * s)) >> x;
                        if (c & 1u) mbar_wait_bounded(&full[s][x], (c >> 8) & 1u, 1u << 26, kWaitNs / 1000);
                    }
            }
        } else {
            // Publisher of the CTA's row blocks (role 1) or column blocks (role 2), in the order in
            // which the panels store them: a block's flag follows the four warps that store it. The
            // progress key of the row's t-th block in round k is k * (CB + 1) + t + 1; of the
            // column's block, k + 1.
            const bool rows = role == 1;
            const uint32_t* prog = rows ? prog_row : prog_col;
            const int k0 = rows ? 2 * I : 2 * J * CB, k1 = min(NR, rows ? k0 + 2 : k0 + 2 * CB), n = rows ? nc : 1;
            for (int k = k0; k < k1; ++k) {
                const int h = k & 1;
                // The warps of row half h are 4h .. 4h + 3; those of column half h are 0 2 5 7 or 1 3 4 6.
                const int w = rows ? 4 * h + (lane & 3) : ((lane & 3) < 2 ? 2 * (lane & 3) + h : 2 * (lane & 3) + 1 - h);
                const int t0 = rows ? first_col(k) : 0;
                for (int t = 0; t < n; ++t) {
                    const int x = t0 + t < n ? t0 + t : t0 + t - n;
                    const uint32_t key = rows ? uint32_t(k) * (CB + 1) + uint32_t(t) + 1u : uint32_t(k) + 1u;
                    const uint64_t since = global_ns();
                    bool ok = true;
                    for (uint32_t it = 1; !__all_sync(0xFFFFFFFFu, ld_acquire_smem(prog + w) >= key); ++it) {
                        const bool late = P.wait_ns == 0u || ((it & 255u) == 0u && global_ns() - since > 4 * P.wait_ns);
                        if (__any_sync(0xFFFFFFFFu, late)) {
                            ok = false;
                            break;
                        }
                        __nanosleep(200);  // the compute warps need the issue slots (1 % of a call against 40 ns)
                    }
                    if (!ok) {
                        raise_device_error(P.words + kWordErr, kErrTmaTimeout);
                        return;
                    }
                    __syncwarp();
                    if (lane == 0) {
                        __threadfence();
                        fence_proxy_async_all();
                        st_release_gpu(rows ? P.flag_b + k * NB + J * CB + x : P.flag_a + k * NB + I, 1u);
                    }
                    __syncwarp();
                }
            }
        }
        return;
    }

    // ---- Compute warps. ----
    const int rg = warp >> 1, ch = (warp & 1) ^ (warp >> 2), rh = rg >> 1;  // row group, column and row half
    const int pair = 2 * rh + ch;
    const int tr = rg * 4 + (lane >> 3), tc = ch * 8 + (lane & 7);
    const int lr = tr & 7, lc = tc & 7;   // within a 32 x 32 piece
    const int lt = (rg & 1) * 32 + lane;  // among the 64 threads of a piece
    uint32_t c[CB][QR][QC];
    uint32_t base = P.base;
    {
        const bool vec = P.ld % 4 == 0 && (reinterpret_cast<uintptr_t>(P.d) & 15) == 0;
        uint32_t lo = 0xFFFFFFFFu, hi = 0u;
        bool over = false;
        auto load = [&]() {
#pragma unroll
            for (int y = 0; y < CB; ++y) load_defeats<LB>(c[y], P, base, I, J * CB + y, tr, tc, vec, lo, hi, over);
        };
        load();
        if (P.automatic) {
            // Every CTA adds its range, waits for all of them, and takes the same decision.
            for (int o = 16; o; o >>= 1) {
                lo = min(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, o));
                hi = max(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
            }
            if (lane == 0 && hi != 0u) {
                atomicMin(&s_lo, lo);
                atomicMax(&s_hi, hi);
            }
            sync_compute();
            if (tid == 0) {
                if (s_hi != 0u) {
                    atomicMax(P.words + kWordLo, ~s_lo);  // the area starts at zero
                    atomicMax(P.words + kWordHi, s_hi);
                }
                if (!all_here(P.words + kWordArrived, gridDim.x, P.start_ns)) {
                    s_go = 0u;
                } else {
                    const uint32_t ghi = ld_acquire_gpu(P.words + kWordHi), glo = ~ld_acquire_gpu(P.words + kWordLo);
                    if (ghi > 0xFFFFu) {
                        if (ghi - glo < 0xFFFFu) s_base = glo - 1u;
                        else s_go = 0u;
                        if (!s_go && blockIdx.x == 0) P.words[kWordWide] = 1u;
                    }
                }
            }
        } else if (LB == 16 && over) {
            atomicOr(P.words + kWordOverflow, 1u);
        }
        __syncthreads();  // with the helper warps
        if (!s_go) return;
        if (s_base != base) {
            base = s_base;
            load();
        }
    }

    bool dead = false;  // a wait of this thread ran out: it waits no more
    auto gave_up = [&]() {
        s_dead = 1u;
        dead = true;
    };
    auto wait_slot = [&](int k, int x) __attribute__((always_inline)) {
        if (!dead && !mbar_wait_bounded(&full[k % kStages][x], uint32_t(k / kStages) & 1u, P.polls, 2 * P.wait_ns))
            gave_up();
    };
    auto wait_b = [&](int k) __attribute__((always_inline)) {
#pragma unroll
        for (int y = 0; y < CB; ++y) wait_slot(k, 1 + y);
    };
    // Every warp is done with the round that used k's stage before.
    auto wait_free = [&](int k) __attribute__((always_inline)) {
        if (!dead && k >= kStages &&
            !mbar_wait_bounded(&empty[k % kStages], uint32_t(k / kStages - 1) & 1u, P.polls, 2 * P.wait_ns))
            gave_up();
    };
    // A block's cells out of and back into the tile (y is uniform, the registers are static).
    uint32_t w[QR][QC];
    auto get = [&](int cb) __attribute__((always_inline)) {
#pragma unroll
        for (int y = 0; y < CB; ++y)
            if (cb == y) {
#pragma unroll
                for (int r = 0; r < QR; ++r)
#pragma unroll
                    for (int q = 0; q < QC; ++q) w[r][q] = c[y][r][q];
            }
    };
    auto put = [&](int cb) __attribute__((always_inline)) {
#pragma unroll
        for (int y = 0; y < CB; ++y)
            if (cb == y) {
#pragma unroll
                for (int r = 0; r < QR; ++r)
#pragma unroll
                    for (int q = 0; q < QC; ++q) c[y][r][q] = w[r][q];
            }
    };
    uint32_t* const dt = smem + SL::DT;  // [k & 1]: D of round k in A form, and in B form
    uint32_t* const db = smem + SL::DB;
    uint32_t* const pair_a = smem + SL::PAIR_A;  // [pair]
    uint32_t* const pair_b = smem + SL::PAIR_B;
    uint32_t* const side_a = smem + SL::SIDE_A;
    uint32_t* const side_b = smem + SL::SIDE_B;
    ChainBuf<LB>& chain = *reinterpret_cast<ChainBuf<LB>*>(smem + SL::CHAIN);
    const int at_a = 4 * lc * kP + 4 * lr, at_b = 4 * lr * WH + QC * lc;  // this thread's cells of a piece
    auto mail = [&](int k, int box) { return P.mail + int64_t(k >> 1) * G::MAIL + box; };
    auto mail_a = [&](int k) { return mail(k, G::MAIL_A) + (k & 1) * 128 * G::QW; };
    auto mail_b = [&](int k) { return mail(k, G::MAIL_B) + (k & 1) * 128 * G::QW; };
    const bool diag_only = 2 * I < NR && in_cols(2 * I) && nc == 1;  // its diagonal block is all that this CTA has
    // The pieces of 64 threads in box and, if box2, box2, into w and w2.
    uint32_t w2[QR][QC];
    auto recv = [&](const uint64_t* box, const uint64_t* box2) __attribute__((always_inline)) {
        bool have = false, have2 = box2 == nullptr;
        uint64_t t0 = 0;
        for (uint32_t it = 0; !dead; ++it) {
            if (!have) have = poll_piece<LB>(w, box, lt);
            if (!have2) have2 = poll_piece<LB>(w2, box2, lt);
            if (have && have2) break;
            if ((it & 255u) == 0u) {
                const uint64_t now = global_ns();
                if (P.wait_ns == 0u) gave_up();
                else if (it == 0) t0 = now;
                else if (now - t0 > P.wait_ns) gave_up();
            }
        }
    };
    auto keep_d = [&](int k) __attribute__((always_inline)) {
        store_a<LB, kP>(w, dt + (k & 1) * G::PA_WORDS + at_a);
        store_b<LB, WH>(w, db + (k & 1) * G::PB_WORDS + at_b);
    };
    auto close_and_send = [&](int k) __attribute__((always_inline)) {
        close_piece<LB>(w, lr, lc, pivots(k), chain, pair);
        send_piece<LB>(w, mail(k, G::MAIL_D) + (k & 1) * 64 * G::QW, lt);
        keep_d(k);
    };
    auto recv_d = [&](int k) __attribute__((always_inline)) {
        recv(mail(k, G::MAIL_D) + (k & 1) * 64 * G::QW, nullptr);
        keep_d(k);
    };

    // The diagonal block of rounds k and k + 1 (k even), in its owner. Each pair brings its piece up
    // to date with rounds k - 2 and k - 1, by mail; (0, 0) closes D; (0, 1) and (1, 0) take their part of round k's row
    // and column panel; (1, 1) takes round k from them and closes D of round k + 1. Each CTA does
    // this at most once, so no buffer or barrier here is used twice.
    auto diagonal = [&](int k) __attribute__((always_inline)) {
        uint32_t* const pa = pair_a + pair * G::PA_WORDS;
        uint32_t* const pb = pair_b + pair * G::PB_WORDS;
        for (int q = kEarly ? k - 2 : k - 1; q < k; ++q) {
            if (q < 0) continue;
            const bool own_a = in_cols(q);  // that column panel is this CTA's
            recv(mail_b(q) + ch * 64 * G::QW, own_a ? nullptr : mail_a(q) + rh * 64 * G::QW);
            store_b<LB, WH>(w, pb + at_b);
            if (own_a) wait_slot(q, 0);
            else store_a<LB, kP>(w2, pa + at_a);
            sync_pair(pair);
            get(col_of(k));
            if (own_a) relax_block<LB, kB, WH>(w, slot_a(q) + 4 * tr, pb + QC * lc, kP);
            else relax_block<LB, kP, WH>(w, pa + 4 * lr, pb + QC * lc, kP);
            put(col_of(k));
            sync_pair(pair);
        }
        get(col_of(k));
        if (pair == 0) {
            close_and_send(k);
            arrive_threads<192>(kBarD);
        } else if (pair == 1) {
            store_b<LB, WH>(w, pb + at_b);
            sync_threads<192>(kBarD);
            relax_block<LB, kP, WH>(w, dt + 4 * lr, pb + QC * lc, pivots(k));
            send_piece<LB>(w, mail(k, G::MAIL_SIDE_B), lt);
            sync_pair(pair);
            store_b<LB, WH>(w, pb + at_b);
            arrive_threads<192>(kBarSides);
        } else if (pair == 2) {
            store_a<LB, kP>(w, pa + at_a);
            sync_threads<192>(kBarD);
            relax_block<LB, kP, WH>(w, pa + 4 * lr, db + QC * lc, pivots(k));
            send_piece<LB>(w, mail(k, G::MAIL_SIDE_A), lt);
            sync_pair(pair);
            store_a<LB, kP>(w, pa + at_a);
            arrive_threads<192>(kBarSides);
        } else {
            sync_threads<192>(kBarSides);
            relax_block<LB, kP, WH>(w, pair_a + 2 * G::PA_WORDS + 4 * lr, pair_b + G::PB_WORDS + QC * lc, pivots(k));
            if (k + 1 < NR) close_and_send(k + 1);
        }
        put(col_of(k));
    };
    // The CTA's row panel of round k, by the four warps that hold its rows: round k - 1 on them, then
    // the product with D. The blocks are stored for the other CTAs in the publisher's order; the
    // pieces that the next diagonal block waits for are mailed first.
    auto row_panel = [&](int k) __attribute__((always_inline)) {
        const int h = k & 1;
        const bool diag = in_cols(k);
        const int y0 = first_col(k);
        const bool send = next_col(k) >= 0 && next_col(k) < nc;
        // Round k - 1's column operand of these rows. In an odd round that round is this block's first:
        // its rows are this CTA's B slots, its column piece comes from the diagonal block's owner.
        const uint32_t* const side = (diag ? pair_a + 2 * G::PA_WORDS : side_a) + 4 * lr;
        const bool apply = k > 0 && !diag_only;
        if (apply && h == 1 && !diag) {
            if (ch == 1) {
                recv(mail(k - 1, G::MAIL_SIDE_A), nullptr);
                store_a<LB, kP>(w, side_a + at_a);
            }
            sync_rows(h);
        }
        if (apply && h == 0) wait_slot(k - 1, 0);
        auto to_slot = [&](const uint32_t(&v)[QR][QC], int y) {
            store_b<LB, G::WPB>(v, slot_b(k, y) + 4 * lr * G::WPB + QC * tc);
        };
        if (apply) {
            wait_b(k - 1);
            if (h == 1) relax_row<LB, CB, kP, G::WPB>(c, side, slot_b(k - 1, 0) + QC * tc, kP);
            else relax_row<LB, CB, kB, G::WPB>(c, slot_a(k - 1) + 4 * tr, slot_b(k - 1, 0) + QC * tc, kP);
        }
        wait_free(k);
#pragma unroll
        for (int y = 0; y < CB; ++y)
            if (y < nc) to_slot(c[y], y);
        if (!diag && ch == h) recv_d(k);
        sync_rows(h);
        relax_row<LB, CB, kP, G::WPB>(c, dt + h * G::PA_WORDS + 4 * lr, slot_b(k, 0) + QC * tc, pivots(k));
        if (send && (h == 1 || kEarly)) {
            get(y0);
            send_piece<LB>(w, mail_b(k) + ch * 64 * G::QW, lt);
        }
        sync_rows(h);  // the slots' first contents are read
#pragma unroll
        for (int y = 0; y < CB; ++y)
            if (y < nc) to_slot(c[y], y);
        sync_rows(h);
        if (warp == (h ? 5 : 0) && lane == 0 && !dead) {
            for (int y = 0; y < nc; ++y) mbar_arrive(&full[k % kStages][1 + y]);
        }
        for (int t = 0; t < nc; ++t) {
            const int y = y0 + t < nc ? y0 + t : y0 + t - nc;
            get(y);
            store_b<LB, G::WPB>(w, block_b(k, y) + 4 * lr * G::WPB + QC * tc);
            __syncwarp();
            if (lane == 0) st_release_smem(&prog_row[warp], uint32_t(k) * (CB + 1) + uint32_t(t) + 1u);
        }
    };
    // The CTA's column panel of round k, by the four warps that hold its columns. In the diagonal
    // block's owner, diagonal() has brought the cells up to date and, in the first round, finished them.
    auto col_panel = [&](int k) __attribute__((always_inline)) {
        const int cb = col_of(k), h = k & 1;
        const bool diag = in_rows(k);
        if (!diag && h == 1) {
            if (rh == 1) {
                recv(mail(k - 1, G::MAIL_SIDE_B), nullptr);
                store_b<LB, WH>(w, side_b + at_b);
            }
            sync_cols(h);
            wait_slot(k - 1, 0);  // this CTA's column panel of round k - 1
            get(cb);
            relax_block<LB, kB, WH>(w, slot_a(k - 1) + 4 * tr, side_b + QC * lc, kP);
        } else if (!diag && k > 0) {
            wait_slot(k - 1, 0);
            wait_slot(k - 1, 1 + cb);
            get(cb);
            relax_block<LB, kB, G::WPB>(w, slot_a(k - 1) + 4 * tr, slot_b(k - 1, cb) + QC * tc, kP);
        } else {
            get(cb);
        }
        wait_free(k);
        uint32_t* const slot = slot_a(k) + 4 * lc * kB + 4 * tr;
        store_a<LB, kB>(w, slot);
        if (!diag || h == 1) {
            put(cb);
            if (!diag && rh == h) {
                recv_d(k);
                get(cb);
            }
            sync_cols(h);
            relax_block<LB, kB, WH>(w, slot_a(k) + 4 * tr, db + h * G::PB_WORDS + QC * lc, pivots(k));
            if ((h == 1 || kEarly) && I == (k >> 1) + 1 && (k >> 1) + 1 >= (J + 1) * CB)  // the next diagonal block is another CTA's
                send_piece<LB>(w, mail_a(k) + rh * 64 * G::QW, lt);
            put(cb);
            sync_cols(h);  // the slot's first contents are read
            store_a<LB, kB>(w, slot);
        }
        sync_cols(h);
        if (warp == h && lane == 0 && !dead) mbar_arrive(&full[k % kStages][0]);
        store_a<LB, kB>(w, block_a(k) + 4 * lc * kB + 4 * tr);
        __syncwarp();
        if (lane == 0) st_release_smem(&prog_col[warp], uint32_t(k) + 1u);
    };
    // Per round: this warp's part of the next round's panels; the diagonal block, two rounds ahead of
    // its own (so that it waits for mail, not for the published blocks of the two rounds before);
    // and the rest of the round: all but the rows that a row panel has taken.
    if (I == 0 && J == 0) diagonal(0);
#pragma unroll 1
    for (int k = -1; k < NR; ++k) {
        const int h = k & 1;
        if (!kEarly && h == 1 && k > 0 && in_rows(k + 1) && in_cols(k + 1)) diagonal(k + 1);
        if (in_rows(k + 1) && rh != h) row_panel(k + 1);
        if (in_cols(k + 1) && ch != h) col_panel(k + 1);
        if (k < 0) continue;
        if (kEarly && h == 0 && in_rows(k + 2) && in_cols(k + 2)) diagonal(k + 2);
        const bool taken = (in_rows(k) && rh == h) || (in_rows(k + 1) && rh != h) ||
                           (diag_only && k >= 2 * I - (kEarly ? 2 : 1) && k <= 2 * I);
        // No warp leaves a round before its slots are filled, so the producer is never lapped.
        wait_slot(k, 0);
        wait_b(k);
        if (!taken) relax_row<LB, CB, kB, G::WPB>(c, slot_a(k) + 4 * tr, slot_b(k, 0) + QC * tc, pivots(k));
        // This thread's slot writes come before the copies that follow.
        if (in_rows(k) || in_cols(k) || in_rows(k + 1) || in_cols(k + 1)) fence_proxy_async_all();
        __syncwarp();
        if (lane == 0 && !dead) mbar_arrive(&empty[k % kStages]);
    }

    if (dead) raise_device_error(P.words + kWordErr, kErrTmaTimeout);
    arrive_threads<kNT + 32>(kBarEnd);

    // Output: widened, shifted back, zero on the diagonal (the reference's masks).
    const bool vec_out = P.ld_out % 4 == 0 && (reinterpret_cast<uintptr_t>(P.out) & 15) == 0;
#pragma unroll
    for (int y = 0; y < CB; ++y)
#pragma unroll
        for (int r = 0; r < QR; ++r) {
            const int i = I * kB + 4 * tr + r, j0 = (J * CB + y) * kB + 4 * tc;
            uint32_t v[4];
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const uint32_t word = c[y][r][n / G::CPW];
                v[n] = LB == 16 ? (word >> (16 * (n % G::CPW))) & 0xFFFFu : word;
                if (LB == 16 && v[n]) v[n] += base;
                if (i == j0 + n) v[n] = 0u;
            }
            if (i < P.C) {
                uint32_t* o = P.out + int64_t(i) * P.ld_out + j0;
                if (vec_out && j0 + 4 <= P.C) {
                    st4(o, v);
                } else {
#pragma unroll
                    for (int n = 0; n < 4; ++n)
                        if (j0 + n < P.C) o[n] = v[n];
                }
            }
        }
}

// ------------------------------------------------------------------------------------------
// Host side.
// ------------------------------------------------------------------------------------------
struct Shape {
    int cb, occ;  // blocks per CTA, CTAs per SM
    const void* fn;
    int smem;
};

template <int LB, int CB, int OCC, int ST> Shape shape() {
    return {CB, OCC, reinterpret_cast<const void*>(resident_kernel<LB, CB, OCC, ST>), smem_layout<LB, CB, ST>::BYTES};
}

// Shapes from the smallest tile to the largest; a matrix takes the first whose CTAs all fit the GPU.
// Fewer blocks per CTA leave a panel less work between two steps of the chain. One B200, se_closure,
// us (blocks per CTA x CTAs per SM; last the launches of closure.cu):
//   16-bit lanes   C = 768    1x1 159   1x2 172   2x1 218   2x2 253   launches 329
//                  C = 1024             1x2 230   2x1 282   2x2 309   launches 429
//                  C = 1344                       3x1 442   2x2 433   launches 612
//                  C = 1500             4x1 586   2x2 487   3x2 596   launches 694
//                  C = 2048                       3x2 966   4x2 1028  launches 950: not taken
//   32-bit lanes   C = 1024             1x2 329   2x1 373             launches 593
//                  C = 1344                       3x1 610   2x2 820   launches 777
//                  C = 1500                       4x1 879             launches 866: not taken
// The shapes taken, with the check-in, against the launches (a whole call): 16-bit lanes C = 16 50 / 67, 64 52 / 66,
// 65 62 / 67, 128 63 / 66, 129 66 / 105, 256 81 / 134, 512 118 / 228, 768 156 / 324, 1024 220 / 423, 1088 237 /
// 481, 1344 418 / 602, 1536 489 / 700; 32-bit lanes C = 16 43 / 71, 64 53 / 71, 128 68 / 71, 129 70 / 134, 256
// 95 / 184, 512 156 / 322, 768 217 / 457, 1024 325 / 589, 1344 612 / 770.
// Two CTAs per SM take no more than 80 registers a thread, and in 32-bit lanes three stages. All shapes but
// the first spill a little (stores / loads, bytes: 16-bit 1x2 48 / 104, 2x2 76 / 176; 32-bit 1x1 40 / 96, 1x2
// 232 / 556, 3x1 112 / 348): the helper warps' registers are allocated at the compute warps' count.
const Shape* shapes(int lane_bits, int* n) {
    static const Shape s16[] = {shape<16, 1, 1, 4>(), shape<16, 1, 2, 4>(), shape<16, 2, 2, 4>()};
    static const Shape s32[] = {shape<32, 1, 1, 4>(), shape<32, 1, 2, 3>(), shape<32, 3, 1, 4>()};
    *n = 3;
    return lane_bits == 16 ? s16 : s32;
}

int64_t ctas(const Shape& s, int64_t NB) { return NB * ((NB + s.cb - 1) / s.cb); }

const Shape* choose(int C, int lane_bits, int sms) {
    const int64_t NB = (int64_t(C) + kB - 1) / kB;
    int n = 0;
    const Shape* s = shapes(lane_bits, &n);
    for (int i = 0; i < n; ++i)
        if (ctas(s[i], NB) <= int64_t(sms) * s[i].occ) return s + i;
    return nullptr;
}

// [0, 256): flags words; then the block flags and the mailboxes (all zeroed per call); then A and B.
struct Layout {
    int64_t NB, NR, flag_a, flag_b, mail, zero_bytes, a, b, total;
};
Layout layout_of(int C, int lane_bits) {
    Layout L;
    L.NB = (int64_t(C) + kB - 1) / kB;
    L.NR = (int64_t(C) + kP - 1) / kP;
    const int64_t blocks = L.NR * L.NB;
    L.flag_a = 256;
    L.flag_b = L.flag_a + blocks * 4;
    L.mail = round_up(L.flag_b + blocks * 4, 256);
    L.zero_bytes = L.mail + L.NB * (lane_bits == 16 ? geo<16>::MAIL : geo<32>::MAIL) * 8;
    L.a = round_up(L.zero_bytes, 1024);
    L.b = L.a + blocks * kP * kB * 4;
    L.total = L.b + blocks * kP * kB * (lane_bits == 16 ? 2 : 4);
    return L;
}

int64_t workspace_bytes(int C, int lane_bits) {
    if (C < 1 || C > max_candidates(lane_bits)) return 0;
    return layout_of(C, lane_bits).total;
}

// The resident launches of a device that may still be in flight, one entry per stream. Two of them that
// do not fit the GPU together could each hold part of the SMs until both give way, so a launch that does
// not fit beside those of other streams is not made: the closure then runs as launches. Nothing ever
// waits for another stream. Streams and contexts are told apart by their ids: a handle may be
// another thread's stream (cudaStreamPerThread), or a new stream in place of a destroyed one.
struct Flight {
    unsigned long long ctx = 0, stream = 0;
    cudaEvent_t done = nullptr;  // of ctx; after the last launch of a call that only queues
    int ctas = 0;                // of the largest launch not known to be done; 0: a free entry
    int held = 0;                // calls that have not let go of the entry yet (Hold)
};
constexpr int kMaxFlights = 32;  // streams; with more in flight a closure runs as launches
struct Flights {
    std::mutex m;
    Flight f[kMaxFlights];
};
constexpr int kMaxDevices = 64;
Flights& flights_of(int dev) {
    static Flights all[kMaxDevices];
    return all[dev];
}

// An event may be asked for while another thread captures a stream.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// Frees the entries whose event has come. A call that waits needs no event, and one whose launch fits
// asks for none, so this costs only those that would have to run as launches.
void drop_finished(Flights& F, unsigned long long ctx) {
    RelaxedCapture relaxed;
    for (Flight& x : F.f)
        if (x.ctas && x.held == 0 && x.ctx == ctx) {
            const cudaError_t e = x.done ? cudaEventQuery(x.done) : cudaSuccess;
            if (e == cudaSuccess) x.ctas = 0;
            else if (e == cudaErrorNotReady) cudaGetLastError();
        }
}

// The entry under which a launch of that many CTAs may be made, or null where it does not fit. A CTA
// is counted as a whole SM, wherever it lands: CTAs that add up to no more than the SMs find room.
Flight* admit(Flights& F, unsigned long long ctx, unsigned long long stream, int ctas, int sms, bool queued) {
    std::lock_guard<std::mutex> lock(F.m);
    for (int pass = 0; pass < 2; ++pass) {
        if (pass) drop_finished(F, ctx);
        Flight *mine = nullptr, *spare = nullptr;
        int others = 0;
        for (Flight& x : F.f) {
            if (x.held == 0 && (x.ctas == 0 || x.ctx != ctx)) {  // another context's may be gone with it
                if (!spare || x.ctas == 0) spare = &x;
            } else if (x.ctx == ctx && x.stream == stream) {
                mine = &x;
            } else if (x.ctx == ctx) {
                others += x.ctas;
            }
        }
        Flight* x = mine ? mine : spare;
        if (!x || (others && others + ctas > sms)) continue;
        if (x != mine) {
            if (x->ctx != ctx) x->done = nullptr;  // neither asked for nor reused
            x->ctx = ctx;
            x->stream = stream;
            x->ctas = 0;
        }
        if (queued && !x->done && cudaEventCreateWithFlags(&x->done, cudaEventDisableTiming) != cudaSuccess) {
            cudaGetLastError();
            x->done = nullptr;
            return nullptr;
        }
        x->ctas = std::max(x->ctas, ctas);
        ++x->held;
        return x;
    }
    return nullptr;
}

Hold::~Hold() {
    if (!flight) return;
    std::lock_guard<std::mutex> lock(static_cast<Flights*>(flights)->m);
    Flight& x = *static_cast<Flight*>(flight);
    // The call has waited for its stream. (Where another thread queued on that stream meanwhile, its launch is
    // no longer counted; two launches that then do not fit together settle it by the check-in.)
    if (--x.held == 0 && !queued) x.ctas = 0;
}

// The check-in's limit, of the calling thread's launches. Once the CTAs that there is room for spin, the
// time is lost to everyone, so it is about what the launches take longer than the resident form
// (0.1 to 0.3 ms); CTAs that find room come within some 10 us, so this limit is for other kernels to end.
constexpr uint64_t kStartNs = 1000000ull;
thread_local uint64_t g_start_ns = kStartNs;
void set_start_limit(uint64_t ns) { g_start_ns = ns; }
thread_local uint64_t g_wait_ns = kWaitNs;
void set_wait_limit(uint64_t ns) { g_wait_ns = std::min(ns, 5 * kWaitNs); }

se_status_t run(const uint32_t* d, int64_t ld, int C, uint32_t* out, int64_t ld_out, int lane_bits, uint32_t base,
                bool automatic, void* d_work, int64_t work_bytes, cudaStream_t s, Hold& hold, bool* ran) {
    *ran = false;
    if (C > max_candidates(lane_bits) || work_bytes < workspace_bytes(C, lane_bits)) return SE_OK;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    SE_CUDA_TRY(cudaStreamIsCapturing(s, &cap));
    if (cap != cudaStreamCaptureStatusNone) return SE_OK;  // replays are not ordered against one another
    int dev = 0, sms = 0, coop = 0;
    SE_CUDA_TRY(cudaGetDevice(&dev));
    SE_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    SE_CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    const Shape* sh = coop && dev < kMaxDevices ? choose(C, lane_bits, sms) : nullptr;
    if (!sh) return SE_OK;
    if (se_status_t st = raise_smem_limit(sh->fn, sh->smem, "the resident closure")) return st;

    const Layout L = layout_of(C, lane_bits);
    uint8_t* work = static_cast<uint8_t*>(d_work);
    Params P;
    P.d = d;
    P.ld = ld;
    P.out = out;
    P.ld_out = ld_out;
    P.words = reinterpret_cast<uint32_t*>(work);
    P.flag_a = reinterpret_cast<uint32_t*>(work + L.flag_a);
    P.flag_b = reinterpret_cast<uint32_t*>(work + L.flag_b);
    P.mail = reinterpret_cast<uint64_t*>(work + L.mail);
    P.A = reinterpret_cast<uint32_t*>(work + L.a);
    P.B = reinterpret_cast<uint32_t*>(work + L.b);
    P.C = C;
    P.NB = int(L.NB);
    P.NR = int(L.NR);
    P.tiles_j = int((L.NB + sh->cb - 1) / sh->cb);
    P.base = base;
    P.automatic = automatic ? 1 : 0;
    P.start_ns = g_start_ns;
    P.wait_ns = g_wait_ns;
    P.polls = P.wait_ns ? 1u << 26 : 1u;

    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(ctas(*sh, L.NB)));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = size_t(sh->smem);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* args[] = {&P};
    unsigned long long stream_id = 0;
    SE_CUDA_TRY(cudaStreamGetId(s, &stream_id));
    Flights& F = flights_of(dev);
    Flight* flight = admit(F, current_context_id(), stream_id, int(cfg.gridDim.x), sms, hold.queued);
    if (!flight) return SE_OK;
    hold.flights = &F;
    hold.flight = flight;
    SE_CUDA_TRY(cudaMemsetAsync(work, 0, size_t(L.zero_bytes), s));
    const cudaError_t e = cudaLaunchKernelExC(&cfg, sh->fn, args);
    if (e == cudaErrorCooperativeLaunchTooLarge) {  // fewer CTAs fit than on a whole B200
        cudaGetLastError();
        return SE_OK;
    }
    SE_CUDA_TRY(e);
    if (hold.queued) SE_CUDA_TRY(cudaEventRecord(flight->done, s));
    *ran = true;
    return SE_OK;
}

}  // namespace resident
}  // namespace se
