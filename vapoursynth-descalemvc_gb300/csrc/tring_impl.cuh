// Chunk-delayed transposing kernels with the sample ring in tensor memory:
// the two passes of a Float32 2D descale.
//
// Both passes read vectors whose samples are adjacent (rows of the input
// plane; columns of the intermediate) and write their results transposed,
// destination-major with the vectors adjacent.  A lane owns V vectors, a warp
// 32 V.
//
//  * Loads: blocks of 128 bytes of every vector of the warp come by TMA (one
//    tensor map per plane, 128-byte swizzle) into one of the warp's two
//    staging buffers, completed on that buffer's mbarrier; the next block is
//    in flight while the current one is consumed.  The swizzle lets a lane
//    read its own vectors without bank conflicts.  Every wait is bounded.  Rows
//    that no tensor map admits come word by word (copy_words).
//  * Ring: a lane converts 16 samples of its vectors at a time to float and
//    stores them to tensor memory (lane = vector, column = sample mod 48, the
//    first 16 columns again after the ring so that every window of up to 16
//    is contiguous).  A destination's window is then one load at a column
//    that is known only at run time: tensor memory serves as a register file
//    that can be indexed, at about 1.3 SM cycles for 8 columns of a warp,
//    where shared memory takes 8 (and the sample scatter 1.5 a sample).
//  * Forward values: also in tensor memory, two chunks a vector, so that the
//    substitutions are loops over groups of destinations instead of 32
//    unrolled destinations on 64 registers of forward values; ring and
//    forward values are 128 columns, four CTAs of one vector a lane an SM.
//  * Intermediate: in tiles of 32 rows, [row / 32][destination][row mod 32]:
//    the first pass stores at constant offsets, the second reads 128
//    contiguous bytes of each vector.
//  * One-axis passes (RingLayout rows, columns): a row's 32 results of a chunk
//    go to shared memory in the output map's swizzle and out by TMA, a
//    column's samples come in boxes of 32 rows.  Their gather keeps the
//    reference CUDA order.  Measured on one GB300, eight 1080p Float32 planes
//    (one thread a vector, uncoalesced stores, before): rows to 1440 508 ->
//    49 us, columns to 810 lines 381 -> 47 us.
//  * Records: copied (cp.async) a chunk of 32 destinations at a time, three
//    deep, for the CTA's four warps.  A warp-wide load of the same 16 bytes
//    takes two shared-memory cycles, which is what two vectors a lane save.
//  * Arithmetic: exact forward substitution (the gather's even and odd taps
//    in two sums), chunk-delayed backward substitution with a zero-carry
//    warm-up over the following chunk.  Every rounding is the same for any V.
//
// What bounds them: instruction issue and dependent FMA chains (43-50 % of the
// slots busy at two vectors a lane, 56-64 % on the busiest SM), the shared-memory
// pipe no longer (25-33 %, 70-76 % before).  Measured on one GB300 against the
// kernels with both in registers and shared memory: 64 YUV420P16 1080p frames
// to 810p 769 -> 526 us, 32 4K Float32 frames to 1440p 1017 -> 580 us.
#pragma once

#include "tstream_impl.cuh"

namespace dsmvc_gb {
namespace {

constexpr int kRingThreads = 128;            // four warps: one per tensor-memory lane quarter
constexpr int kRingStep = 16;                // samples converted at a time
// try_wait rounds before a feed wait gives up, each suspending at most
// kFeedWaitSuspendNs (about 65 ms in all, far beyond any copy's latency); a
// stalled warp stops waiting and its kernel reports kStatusFeedStall.
constexpr int kFeedWaitRounds = 1 << 16;
constexpr unsigned kFeedWaitSuspendNs = 1000;
constexpr int kRingBuffers = 2;              // staged blocks: one consumed, the others in flight

// ---- tensor memory -----------------------------------------------------------

__device__ __forceinline__ void tm_ld4(float *x, unsigned a) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]) : "r"(a));
}
__device__ __forceinline__ void tm_ld8(float *x, unsigned a) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]), "=f"(x[4]), "=f"(x[5]), "=f"(x[6]), "=f"(x[7])
                 : "r"(a));
}
__device__ __forceinline__ void tm_st8(unsigned a, const float *x) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};"
                 :: "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]), "f"(x[4]), "f"(x[5]), "f"(x[6]), "f"(x[7]), "r"(a));
}
__device__ __forceinline__ void tm_st4(unsigned a, const float *x) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%4], {%0,%1,%2,%3};"
                 :: "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]), "r"(a));
}
__device__ __forceinline__ void tm_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;"); }
template <int N> __device__ __forceinline__ void tm_ld(float *x, unsigned a) {
#pragma unroll
    for (int i = 0; i + 8 <= N; i += 8) tm_ld8(x + i, a + i);
    if constexpr (N % 8) tm_ld4(x + N / 8 * 8, a + N / 8 * 8);
}
// Every load issued so far has arrived; no use of x moves before this.
template <int N> __device__ __forceinline__ void tm_pin(float *x) {
#pragma unroll
    for (int i = 0; i < N; i += 4)
        asm volatile("" : "+f"(x[i]), "+f"(x[i + 1]), "+f"(x[i + 2]), "+f"(x[i + 3]));
}
__device__ __forceinline__ void tm_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;"); }

// Output samples: rounding before the clamp to [0, out_max] gives what the
// clamp before it does (the bounds are whole, the conversion saturates below
// at 0 and NaN converts to 0).
template <class T> __device__ __forceinline__ T rout(float v, const Conversion &c) {
    if constexpr (sizeof(T) == 4) return v;
    else return static_cast<T>(min(__float2uint_rn(__fadd_rn(__fmul_rn(v, c.out_scale), c.out_offset)), c.out_max));
}

// ---- ring feeder ---------------------------------------------------------------

// Arrivals that complete a block: of vectors that no tensor map admits (not 16-byte
// aligned) every lane copies its words.  A stall test expects one that nothing makes.
template <RingLayout LAYOUT> __device__ __forceinline__ unsigned ring_arrivals(const StreamJob &j, const StreamJob &lead) {
    return (LAYOUT == RingLayout::columns || j.mapped ? 1 : 32) + (lead.feed_stall_test ? 1 : 0);
}

// LAYOUT columns: a vector's samples are a plane's column.
template <class In, int V, int W, RingLayout LAYOUT>
struct RingFeeder {
    static constexpr bool COLS = LAYOUT == RingLayout::columns;
    static constexpr int SPL = 16 / static_cast<int>(sizeof(In));   // samples per 16 bytes
    static constexpr int SB = COLS ? 32 : 8 * SPL;                  // samples per staged block
    static constexpr int DUP = W <= 8 ? 8 : 16;                     // columns stored again after the ring
    static constexpr int VC = kRingColumns + 16;                    // columns per vector
    static constexpr int BUFFER = 32 * V * 128;                     // bytes per staging buffer
    static constexpr int NR = kRingStep * static_cast<int>(sizeof(In)) / 4;   // words of a step's samples

    const StreamJob *job;
    std::uint64_t map;       // the plane's tensor map, 0: vectors not 16-byte aligned
    int first;               // the warp's first vector
    int vectors;             // its valid vectors (>= 1)
    int size;                // samples per vector
    int limit;               // blocks that start before this sample are fetched
    int lane;
    unsigned ring;           // tensor-memory address of the warp's ring
    unsigned stage;          // staging buffers of this warp (shared address)
    unsigned mbar;           // their barriers (8 bytes apart)
    unsigned row[V];         // this lane's vectors in a staging buffer (byte offset)
    float in_offset, in_scale;
    int have;                // samples in the ring (a multiple of 16)
    int column;              // have mod kRingColumns
    int next;                // sample where the next block to fetch starts
    int count;               // blocks consumed or being consumed
    unsigned at;             // the block being consumed (shared address)
    bool tiled;
    bool failed;             // a wait ran out: nothing more is fetched or waited for

    // `stage_at`, `mbar_at`: the warp's staging buffers and their barriers.
    __device__ __forceinline__ void init(const StreamJob &j, int samples, int first_vector, int count_vectors, int l,
                                         unsigned stage_at, unsigned mbar_at) {
        job = &j;
        map = j.mapped ? reinterpret_cast<std::uint64_t>(j.map) : 0;
        first = first_vector;
        vectors = count_vectors;
        size = limit = samples;
        lane = l;
        stage = stage_at;
        mbar = mbar_at;
        // Lanes past the warp's last vector repeat it: same samples, same
        // results, stored to the same place.
#pragma unroll
        for (int a = 0; a < V; ++a) {
            const unsigned v = min(lane + 32 * a, vectors - 1);
            row[a] = COLS ? v * 4 : v * 128 + (v & 7) * 16;
        }
        in_offset = j.conv.in_offset;
        in_scale = j.conv.in_scale;
        tiled = j.mapped == 2;
        failed = false;
        if (map && lane == 0)
            asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;\n" :: "l"(map) : "memory");
        __syncwarp();
    }

    // The block at `next` of `count` vectors from `first` on without a tensor map: a
    // word a lane, 128 contiguous bytes a warp-wide copy, where TMA would put it, zeros
    // past the vectors' end.  By cp.async where the vectors begin at a word.  A lane
    // loading its own vector's next 16 samples, unstaged, waited on memory at each
    // step: one GB300, eight 1919x1079 Float32 planes' rows 219 -> 70 us, sixteen 1079x607
    // planes 67 -> 55, 24 YUV420P8 frames of 720x480 with tight rows 90 -> 81 (a lone frame
    // of 8-bit rows that begin inside a word 23 -> 25: its copies wait), and without
    // those loads in every refill 64 aligned YUV420P16 1080p frames 536 -> 526.
    static __device__ __noinline__ void copy_words(const StreamJob *job, int first, int next, int size, int count,
                                                   unsigned to, unsigned mb) {
        constexpr int PER = 4 / static_cast<int>(sizeof(In));      // samples a word
        const int lane = threadIdx.x & 31, at = next + lane * PER;
        const int samples = max(min(PER, size - at), 0);
        const std::int64_t vec = job->in_vec;
        const In *plane = static_cast<const In *>(job->in);
        const In *p = plane + first * vec + (samples ? at : next);
        auto put = [&](int v) { return to + v * 128 + (((lane >> 2) ^ (v & 7)) * 16) + (lane & 3) * 4; };
        if (PER == 1 || ((reinterpret_cast<std::uint64_t>(plane) | static_cast<std::uint64_t>(vec) * sizeof(In)) & 3) == 0) {
#pragma unroll 8
            for (int v = 0; v < count; ++v, p += vec)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n"
                             :: "r"(put(v)), "l"(p), "r"(samples * static_cast<int>(sizeof(In))) : "memory");
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" :: "r"(mb) : "memory");
        } else {
            // Vectors that begin inside a word: the samples of BATCH in flight
            // at a time, loaded without a branch (repeats past the ends).  Plain
            // loads: the launch before may still write the plane while this
            // one starts.
            constexpr int BATCH = 32 / PER;
            const In *row0 = plane + first * vec;
            int column[PER];
            unsigned mask = 0;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                column[k] = min(at + k, size - 1);
                if (k < samples) mask |= (0xffffffffu >> (32 - 32 / PER)) << (k * 32 / PER);
            }
#pragma unroll 1
            for (int v = 0; v < count; v += BATCH) {
                In x[BATCH][PER];
#pragma unroll
                for (int i = 0; i < BATCH; ++i) {
                    const In *r = row0 + min(v + i, count - 1) * vec;
#pragma unroll
                    for (int k = 0; k < PER; ++k) x[i][k] = r[column[k]];
                }
#pragma unroll
                for (int i = 0; i < BATCH; ++i) {
                    unsigned w = 0;
#pragma unroll
                    for (int k = 0; k < PER; ++k) w |= static_cast<unsigned>(x[i][k]) << (k * 32 / PER);
                    if (v + i < count) asm volatile("st.shared.u32 [%0], %1;\n" :: "r"(put(v + i)), "r"(w & mask) : "memory");
                }
            }
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" :: "r"(mb) : "memory");
        }
    }

    // Fetches the block at `next` into buffer `slot`.
    __device__ __forceinline__ void issue(unsigned slot) {
        if constexpr (!COLS) {
            if (!map) {
                if (next < limit)
                    copy_words(job, first, next, size, vectors, stage + slot * BUFFER, mbar + slot * 8);
                __syncwarp();
                next += SB;
                return;
            }
        }
        unsigned elected;
        asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n selp.u32 %0, 1, 0, q;\n}\n" : "=r"(elected));
        if (elected && next < limit) {
            const unsigned mb = mbar + slot * 8;
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" :: "r"(mb), "r"(BUFFER) : "memory");
            asm volatile("cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes"
                         " [%0], [%1, {%2, %3, %4}], [%5];\n"
                         :: "r"(stage + slot * BUFFER), "l"(map), "r"(COLS ? first : tiled ? 0 : next),
                            "r"(COLS ? next : first), "r"(tiled ? next / 32 : 0), "r"(mb) : "memory");
        }
        next += SB;
    }

    __device__ __forceinline__ bool arrived(int k) const {
        unsigned done;
        asm volatile("{\n .reg .pred q;\n mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2, %3;\n"
                     " selp.u32 %0, 1, 0, q;\n}\n"
                     : "=r"(done) : "r"(mbar + (k & 1) * 8), "r"(k >> 1 & 1), "r"(kFeedWaitSuspendNs) : "memory");
        return done;
    }

    // Waits, within a limit, for the k-th block's copy.
    __device__ __noinline__ bool wait(int k) const {
        for (int it = 0; it < kFeedWaitRounds; ++it)
            if (arrived(k)) return true;
        return false;
    }

    // Enters the next block; the one after it goes to the other buffer, which
    // every lane has read.
    __device__ __forceinline__ void enter() {
        if (!arrived(count) && !failed && !wait(count)) {
            failed = true;
            limit = 0;
        }
        at = stage + (count & 1) * BUFFER;
        ++count;
        __syncwarp();
        issue(count & 1);
    }

    // Waits for the copies still in flight (the block being consumed and the
    // next): none writes to shared memory after the CTA has ended.
    __device__ __forceinline__ void drain() const {
        if (!COLS || map)
            for (int k = max(count - 1, 0), from = next - (count - k + 1) * SB; k <= count; ++k, from += SB)
                if (from < size) wait(k);
    }

    // Loads the next step's samples of every vector.
    __device__ __forceinline__ void fetch(unsigned (&raw)[V][NR]) {
        if (COLS && !map) {
            // Columns that no tensor map admits: each lane loads its own (plain
            // loads: the launch before may still write the plane while this one
            // starts).
#pragma unroll
            for (int a = 0; a < V; ++a) {
                const float *p = static_cast<const float *>(job->in) + first + min(lane + 32 * a, vectors - 1);
                const std::int64_t elem = job->in_elem;
#pragma unroll
                for (int i = 0; i < NR; ++i) raw[a][i] = __float_as_uint(p[min(have + i, size - 1) * elem]);
            }
            return;
        }
        if (have % SB == 0) enter();
        if constexpr (COLS) {
            // [sample][column]: one load a sample.
#pragma unroll
            for (int a = 0; a < V; ++a)
#pragma unroll
                for (int i = 0; i < NR; ++i)
                    asm volatile("ld.shared.u32 %0, [%1];"
                                 : "=r"(raw[a][i]) : "r"(at + row[a] + (have % SB + i) * (128 * V)));
            return;
        }
        // 16-byte pieces lie in the tensor map's 128-byte swizzle.
        const unsigned piece = (have % SB) / SPL;
#pragma unroll
        for (int a = 0; a < V; ++a) {
#pragma unroll
            for (int i = 0; i < NR / 4; ++i)
                asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                             : "=r"(raw[a][4 * i]), "=r"(raw[a][4 * i + 1]), "=r"(raw[a][4 * i + 2]),
                               "=r"(raw[a][4 * i + 3])
                             : "r"(at + (row[a] ^ ((piece + i) * 16))));
        }
    }

    // `from`: a multiple of 16 at most the first window start.
    __device__ __forceinline__ void start(int from, unsigned ring_at) {
        ring = ring_at;
        const float zero[8] = {};
        for (int c = 0; c < V * VC; c += 8) tm_st8(ring + c, zero);
        tm_wait_st();
        have = from;
        column = from % kRingColumns;
        count = 0;
        next = from / SB * SB;
        if (!COLS || map) {
            issue(0);
            if (from % SB) enter();
        }
    }

    // The next 16 samples of every vector.
    __device__ __forceinline__ void step() {
        unsigned raw[V][NR];
        fetch(raw);
#pragma unroll
        for (int a = 0; a < V; ++a) {
            float f[kRingStep];
            if constexpr (sizeof(In) == 4) {
#pragma unroll
                for (int i = 0; i < kRingStep; ++i) f[i] = __uint_as_float(raw[a][i]);
            } else {
                const In *vals = reinterpret_cast<const In *>(raw[a]);
                const float2 off = make_float2(-in_offset, -in_offset), scale = make_float2(in_scale, in_scale);
#pragma unroll
                for (int i = 0; i < kRingStep; i += 2) {
                    const float2 v = make_float2(static_cast<float>(vals[i]), static_cast<float>(vals[i + 1]));
                    const float2 r = __fmul2_rn(__fadd2_rn(v, off), scale);
                    f[i] = r.x;
                    f[i + 1] = r.y;
                }
            }
            const unsigned to = ring + a * VC + column;
            // The ring's first columns are stored again after it (other
            // steps store theirs twice).
            const unsigned dup = column ? to : to + kRingColumns;
#pragma unroll
            for (int i = 0; i < kRingStep; i += 4) {
                tm_st4(to + i, f + i);
                if (i < DUP) tm_st4(dup + i, f + i);
            }
        }
        have += kRingStep;
        column = column + kRingStep == kRingColumns ? 0 : column + kRingStep;
    }

    // Makes samples [0, need) resident (`need`: a multiple of 16, less than 16
    // past the size).
    __device__ __forceinline__ void ensure(int need) {
        if (have >= need) return;
        do step(); while (have < need);
        tm_wait_st();
    }
};

// ---- records ---------------------------------------------------------------------

// Records (StreamPack::ring_forward, ring_backward): per group of four
// destinations, four ring columns (the first word also holds the refill
// target, in blocks of 16 samples, above bit 8), the four inverse diagonals, the four windows' weights,
// and the four destinations' lower factors back to back; the four
// destinations' backward factors back to back.
template <int HB, int W> struct RingRecord {
    static constexpr int LOW = 4 * HB;
    static constexpr int GROUP = 8 + 4 * W + LOW;     // floats per group
    static constexpr int GROUPS = kTChunk / 4;
    static constexpr int CHUNK = GROUPS * (GROUP + LOW);
};

// ---- substitutions ---------------------------------------------------------------

// Destinations per iteration of the substitution loops (each iteration moves
// its histories; one vector a lane spills with more).  Even so half-bandwidth 7 spills
// at one vector (up to 40 bytes stored and 120 loaded a lane).
template <int V> constexpr int kRingGroup = V == 2 ? 16 : 8;

template <int N> __device__ __forceinline__ void rload(float (&c)[N], const float *from) {
    static_assert(N % 4 == 0);
#pragma unroll
    for (int i = 0; i < N; i += 4) {
        const float4 l = tlds4(from + i);
        c[i] = l.x;
        c[i + 1] = l.y;
        c[i + 2] = l.z;
        c[i + 3] = l.w;
    }
}

// Forward substitution of a chunk: store(a, t, y) takes eight values of a
// vector from destination t of the chunk on.  `hist`: the HB values before it,
// oldest first.
// SPLIT: the gather's even and odd taps in two sums, else one after another
// (the reference CUDA order, which one-axis passes keep).
template <int HB, int W, int V, bool SPLIT, class Feed, class Store>
__device__ __forceinline__ void rforward(float (&hist)[V][HB], const float *fwd, Feed &feed, Store &&store) {
    using R = RingRecord<HB, W>;
    constexpr int G = kRingGroup<V>;
#pragma unroll 1
    for (int tg = 0; tg < kTChunk; tg += G) {
        float y[V][HB + G];                               // y[HB + t]: destination tg + t
#pragma unroll
        for (int a = 0; a < V; ++a)
#pragma unroll
            for (int d = 0; d < HB; ++d) y[a][d] = hist[a][d];
#pragma unroll
        for (int t = 0; t < G; t += 4) {
            const float *gr = fwd + ((tg + t) / 4) * R::GROUP;
            const int4 h = *reinterpret_cast<const int4 *>(gr);
            feed.ensure(static_cast<int>(static_cast<unsigned>(h.x) >> 8) * kRingStep);
            const unsigned at[4] = {feed.ring + (h.x & 255), feed.ring + h.y, feed.ring + h.z, feed.ring + h.w};
            float x[2][V][W];
#pragma unroll
            for (int a = 0; a < V; ++a) tm_ld<W>(x[0][a], at[0] + a * Feed::VC);
            float iv[4], lw[R::LOW];
            rload(iv, gr + 4);
            rload(lw, gr + 8 + 4 * W);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                tm_wait_ld();
#pragma unroll
                for (int a = 0; a < V; ++a) tm_pin<W>(x[q & 1][a]);
                if (q < 3) {
#pragma unroll
                    for (int a = 0; a < V; ++a) tm_ld<W>(x[(q + 1) & 1][a], at[(q + 1) & 3] + a * Feed::VC);
                }
                float2 acc[V];
#pragma unroll
                for (int a = 0; a < V; ++a) acc[a] = make_float2(0.0f, 0.0f);
#pragma unroll
                for (int i = 0; i < W; i += 4) {
                    const float4 w = tlds4(gr + 8 + q * W + i);
#pragma unroll
                    for (int a = 0; a < V; ++a) {
                        const float *xa = x[q & 1][a] + i;
                        if constexpr (SPLIT) {
                            acc[a] = __ffma2_rn(make_float2(w.x, w.y), make_float2(xa[0], xa[1]), acc[a]);
                            acc[a] = __ffma2_rn(make_float2(w.z, w.w), make_float2(xa[2], xa[3]), acc[a]);
                        } else {
                            acc[a].x = fmaf(w.y, xa[1], fmaf(w.x, xa[0], acc[a].x));
                            acc[a].x = fmaf(w.w, xa[3], fmaf(w.z, xa[2], acc[a].x));
                        }
                    }
                }
#pragma unroll
                for (int a = 0; a < V; ++a) {
                    float sum = SPLIT ? acc[a].x + acc[a].y : acc[a].x;
#pragma unroll
                    for (int e = 0; e < HB; ++e) sum = fmaf(lw[q * HB + e], y[a][t + q + e], sum);
                    // Records past the end of the vector are zero (inverse
                    // diagonal included): their forward values are zero.
                    y[a][HB + t + q] = sum * iv[q];
                }
            }
        }
#pragma unroll
        for (int a = 0; a < V; ++a) {
#pragma unroll
            for (int t = 0; t < G; t += 8) store(a, tg + t, &y[a][HB + t]);
#pragma unroll
            for (int d = 0; d < HB; ++d) hist[a][d] = y[a][G + d];
        }
    }
}

// Backward substitution of a chunk from its forward values at `ycol` and the
// HB results after it, `carry` (nearest first; the chunk's first HB results
// on return).  MODE 0: the warm-up, nothing stored; 1: every result stored as
// soon as it is known; 2: those of the chunk's first `valid` destinations.
// `at`: the chunk's first destination; STEP: the output's destination stride,
// 0: `out_elem`, -1: rows, whose 32 results of a chunk go to `tile` in shared
// memory (a row of 128 bytes each, in the output map's swizzle).
template <int HB, int W, int V, int MODE, int STEP, class Out>
__device__ __forceinline__ void rbackward(float (&carry)[V][HB], const float *bwd, unsigned ycol, int valid,
                                          Out *const (&out)[V], std::int64_t at, std::int64_t out_elem,
                                          const Conversion &conv, float *tile = nullptr) {
    using R = RingRecord<HB, W>;
    constexpr int G = kRingGroup<V>;
#pragma unroll 1
    for (int tg = kTChunk - G; tg >= 0; tg -= G) {
        float y[V][G], x[V][G + HB];
#pragma unroll
        for (int a = 0; a < V; ++a)
#pragma unroll
            for (int t = 0; t < G; t += 8) tm_ld8(&y[a][t], ycol + a * 2 * kTChunk + tg + t);
#pragma unroll
        for (int a = 0; a < V; ++a)
#pragma unroll
            for (int d = 0; d < HB; ++d) x[a][G + d] = carry[a][d];
        Out *o[V];
        if constexpr (MODE > 0 && STEP >= 0) {
#pragma unroll
            for (int a = 0; a < V; ++a) o[a] = out[a] + (STEP ? (at + tg) * STEP : (at + tg + G - 1) * out_elem);
        }
        float u[2][R::LOW];
        rload(u[(G / 4 - 1) & 1], bwd + (tg / 4 + G / 4 - 1) * R::LOW);
        tm_wait_ld();
#pragma unroll
        for (int a = 0; a < V; ++a) tm_pin<G>(y[a]);
#pragma unroll
        for (int t = G - 1; t >= 0; --t) {
            if (t % 4 == 3 && t > 4) rload(u[(t / 4 - 1) & 1], bwd + (tg / 4 + t / 4 - 1) * R::LOW);
#pragma unroll
            for (int a = 0; a < V; ++a) {
                float sum = 0.0f;
#pragma unroll
                for (int pos = 0; pos < HB; ++pos)
                    sum = fmaf(u[(t / 4) & 1][(t % 4) * HB + pos], x[a][t + (HB == 3 ? pos + 1 : HB - pos)], sum);
                x[a][t] = y[a][t] - sum;
                if constexpr (MODE > 0 && STEP >= 0) {
                    Out *to = STEP ? o[a] + t * STEP : o[a];
                    if (MODE == 1 || tg + t < valid) *to = rout<Out>(x[a][t], conv);
                    if constexpr (STEP == 0) o[a] -= out_elem;
                }
            }
        }
        if constexpr (MODE > 0 && STEP < 0) {
            const int lane = threadIdx.x & 31;
#pragma unroll
            for (int a = 0; a < V; ++a)
#pragma unroll
                for (int t = 0; t < G; t += 4)
                    *reinterpret_cast<float4 *>(tile + (32 * a + lane) * 32 + (((tg + t) / 4) ^ (lane & 7)) * 4) =
                        make_float4(x[a][t], x[a][t + 1], x[a][t + 2], x[a][t + 3]);
        }
#pragma unroll
        for (int a = 0; a < V; ++a)
#pragma unroll
            for (int d = 0; d < HB; ++d) carry[a][d] = x[a][d];
    }
}

// Writes a chunk's rows from `tile`: through the output's tensor map, which
// clips what lies past the plane, or row by row.
template <int V>
__device__ __forceinline__ void rstore_rows(float *tile, std::uint64_t map, float *out, std::int64_t out_vec, int first,
                                            int vectors, int at, int valid) {
    const int lane = threadIdx.x & 31;
    if (map) {
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) {
            asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];\n"
                         :: "l"(map), "r"(at), "r"(first), "r"(0),
                            "r"(static_cast<unsigned>(__cvta_generic_to_shared(tile))) : "memory");
            asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
        }
    } else {
        __syncwarp();
        for (int r = 0; r < vectors; ++r) {
            const float v = tile[r * 32 + ((lane / 4) ^ (r & 7)) * 4 + lane % 4];
            if (lane < valid) out[(first + r) * out_vec + at + lane] = v;
        }
        __syncwarp();
    }
}

// The rows written so far have left `tile`.
__device__ __forceinline__ void rstore_wait() {
    if ((threadIdx.x & 31) == 0) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
    __syncwarp();
}

// Waits for the launch before this one, its results included, where this one
// may start early (RingAhead own, any).  Every thread does: a launch is
// complete only after those before it.
__device__ __forceinline__ void ring_launch_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// Lets such a launch behind this one start once every CTA is past this point (and
// holds its tensor memory).
__device__ __forceinline__ void ring_launch_next() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// A CTA's tensor memory, by its first warp; *base after the next barrier.  Those
// that an allocation waits for wait for nothing: they are past ring_launch_wait, or
// wait behind launches that all hold theirs (RingAhead).
template <int COLUMNS> __device__ __forceinline__ void ring_allocate(unsigned *base, int warp) {
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                     :: "r"(static_cast<unsigned>(__cvta_generic_to_shared(base))), "n"(COLUMNS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
}
__device__ __forceinline__ void ring_allocated() {
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
}

template <int HB, int W, int V, RingLayout LAYOUT, class In, class Out>
__global__ void __launch_bounds__(kRingThreads, 4 / V)
tring_kernel(const StreamJob *__restrict__ jobs, int job_count, bool late) {
    using R = RingRecord<HB, W>;
    using Feed = RingFeeder<In, V, W, LAYOUT>;
    constexpr bool TILED = LAYOUT == RingLayout::tiled, ROWS = LAYOUT == RingLayout::rows;
    constexpr bool SPLIT = LAYOUT == RingLayout::plain || TILED;
    constexpr int LC = kTChunk, WARPS = kRingThreads / 32, STEP = TILED ? 32 : ROWS ? -1 : 0;
    constexpr int COLUMNS = 128 * V;       // the rings and two chunks of forward values
    static_assert(V * (Feed::VC + 2 * LC) <= COLUMNS);
    // Staging buffers (WARPS * kRingBuffers of Feed::BUFFER bytes, where the
    // 128-byte swizzle's pattern of 1024 begins), the rows of a chunk alike,
    // then three chunks of records.
    extern __shared__ unsigned char ring_dynamic[];
    unsigned char *const ring_smem = ring_dynamic + (-static_cast<unsigned>(__cvta_generic_to_shared(ring_dynamic)) & 1023);
    unsigned char *const ring_rows = ring_smem + WARPS * kRingBuffers * Feed::BUFFER;
    float *bufs = reinterpret_cast<float *>(ring_rows + (ROWS ? WARPS * V * 4096 : 0));
    __shared__ unsigned long long feed_bar[WARPS][kRingBuffers];
    __shared__ unsigned tm_base;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // Jobs are assigned warps; a CTA's warps share one plan and one chunk
    // range (the host rounds changes of either up to whole CTAs), whose
    // records the CTA copies once.
    const int cta_warp = static_cast<int>(blockIdx.x) * WARPS;
    const StreamJob &job = jobs[find_tjob(jobs, job_count, cta_warp + warp)];
    const StreamJob &lead = jobs[find_tjob(jobs, job_count, cta_warp)];
    const dev::StreamPlanView p = lead.plan;
    const int n = p.destination_size;
    const int chunks = (n + LC - 1) / LC;
    // Chunks whose outputs this CTA stores: [ca, cb).  The forward
    // substitution runs over [c0, ce]: from `margin` chunks early (zero
    // history) for a range past chunk 0, to one chunk late (the backward warm-up of
    // the last stored chunk) for a range ending before the last chunk.
    const int ca = lead.chunk_begin;
    const int cb = lead.chunk_end > 0 ? lead.chunk_end : chunks;
    const int c0 = max(ca - lead.margin, 0);
    const int ce = cb < chunks ? cb : chunks - 1;

    tstage(bufs + (c0 % 3) * R::CHUNK, p, c0, tid, kRingThreads);
    tcp_commit();
    if (c0 + 1 <= ce) tstage(bufs + ((c0 + 1) % 3) * R::CHUNK, p, c0 + 1, tid, kRingThreads);
    tcp_commit();

    if (!late) ring_allocate<COLUMNS>(&tm_base, warp);
    if (lane < kRingBuffers) {
        const unsigned mb = static_cast<unsigned>(__cvta_generic_to_shared(&feed_bar[warp][lane]));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" :: "r"(mb), "r"(ring_arrivals<LAYOUT>(job, lead)) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    ring_allocated();

    // The warp's vectors; a warp past its job's last vector only takes part
    // in the CTA's record copies and barriers.
    const int warp_first = (cta_warp + warp - job.first_block) * 32 * V;
    const int left = job.vectors - warp_first;
    const bool idle = left <= 0;
    Feed feed;
    feed.init(job, p.source_size, idle ? 0 : warp_first, idle ? 1 : min(left, 32 * V), lane,
              static_cast<unsigned>(__cvta_generic_to_shared(ring_smem + warp * kRingBuffers * Feed::BUFFER)),
              static_cast<unsigned>(__cvta_generic_to_shared(&feed_bar[warp][0])));
    ring_launch_wait();
    if (late) {
        ring_allocate<COLUMNS>(&tm_base, warp);
        ring_allocated();
    }
    const unsigned tm = tm_base;
    if (!idle) feed.start(c0 > 0 ? lead.first_sample : 0, tm + (static_cast<unsigned>(warp * 32) << 16));
    ring_launch_next();

    Out *out[V];
#pragma unroll
    for (int a = 0; a < V; ++a) {
        const int v = idle ? 0 : warp_first + min(lane + 32 * a, feed.vectors - 1);
        out[a] = static_cast<Out *>(job.out) + (TILED ? static_cast<std::int64_t>(v >> 5) * n * 32 + (v & 31) : v);
    }

    const Conversion conv = job.conv;
    const std::int64_t out_elem = job.out_elem;
    float *const tile = reinterpret_cast<float *>(ring_rows + warp * V * 4096);
    const std::uint64_t out_map = ROWS && job.out_mapped ? reinterpret_cast<std::uint64_t>(job.out_map) : 0;
    if (out_map && lane == 0)
        asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;\n" :: "l"(out_map) : "memory");
    // A chunk's rows, once its last results are in `tile`.
    auto rows = [&](int chunk) {
        if constexpr (ROWS)
            rstore_rows<V>(tile, out_map, static_cast<float *>(job.out), job.out_vec, feed.first, feed.vectors, chunk * LC,
                           n - chunk * LC);
    };
    const unsigned ycol = feed.ring + V * Feed::VC;        // chunk c's forward values 32 (c & 1) columns on
    float hist[V][HB], carry[V][HB];
#pragma unroll
    for (int a = 0; a < V; ++a)
#pragma unroll
        for (int d = 0; d < HB; ++d) hist[a][d] = 0.0f;
    for (int c = c0;; ++c) {
        tcp_wait_one();
        __syncthreads();
        const float *cur = bufs + (c % 3) * R::CHUNK;
        float *prev = bufs + ((c + 2) % 3) * R::CHUNK;
        if (!idle) {
            const unsigned yc = ycol + (c & 1) * LC, yp = ycol + (~c & 1) * LC;
            rforward<HB, W, V, SPLIT>(hist, cur, feed, [&](int a, int t, const float *y) { tm_st8(yc + a * 2 * LC + t, y); });
            tm_wait_st();
            const float *cur_b = cur + R::GROUPS * R::GROUP;
#pragma unroll
            for (int a = 0; a < V; ++a)
#pragma unroll
                for (int d = 0; d < HB; ++d) carry[a][d] = 0.0f;
            if (c + 1 == chunks) {
                // The vector's last chunk: exact from the end, stored when the
                // chunk is the CTA's.
                if constexpr (ROWS) rstore_wait();
                rbackward<HB, W, V, 2, STEP>(carry, cur_b, yc, c < cb ? n - c * LC : 0, out, c * LC, out_elem, conv,
                                             tile);
                if (c < cb) rows(c);
            } else if (c > ca) {
                rbackward<HB, W, V, 0, STEP>(carry, cur_b, yc, 0, out, 0, out_elem, conv);
            }
            if (c > ca) {
                if constexpr (ROWS) rstore_wait();
                rbackward<HB, W, V, 1, STEP>(carry, prev + R::GROUPS * R::GROUP, yp, LC, out, (c - 1) * LC, out_elem, conv,
                                             tile);
                rows(c - 1);
            }
        }
        if (c == ce) break;
        // Every warp is done with chunk c-1's records: fetch chunk c+2.
        __syncthreads();
        if (c + 2 <= ce) tstage(prev, p, c + 2, tid, kRingThreads);
        tcp_commit();
    }
    // No copy is left in flight; a stalled feed wait reports.
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    if (!idle) feed.drain();
    if constexpr (ROWS) {
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
    }
    if (__any_sync(0xffffffffu, feed.failed) && lane == 0) atomicOr(lead.status, dev::kStatusFeedStall);
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" :: "r"(tm), "n"(COLUMNS));
}

// Launches behind the launch before it on the stream or, unless that has `ended`,
// while it still ends: the way to the first sample (job table, records, tensor
// memory, barriers), up to 3 us of a pass, then runs beside it.  The kernels
// read only what that launch does not write until ring_launch_wait.  Late
// allocations (RingAhead any) keep some of it back: on the runs measured an SM took no
// second such CTA before the first had allocated.  One Float32 bicubic frame on one
// GB300, frames behind one another, us with each first launch behind the end of the
// frame before, with late and with early allocations: 640x360 20.5, 16.2 and 15.9,
// 1080p 26.7, 23.4 and 20.2, 4K 41.0, 36.4 and 35.5; eight 1080p planes' rows 41.0,
// 35.2 and 33.8.
inline cudaError_t ring_launch(void (*kernel)(const StreamJob *, int, bool), const StreamJob *jobs, int count, int blocks,
                               int smem, RingAhead ahead, cudaStream_t s) {
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(static_cast<unsigned>(blocks));
    config.blockDim = dim3(kRingThreads);
    config.dynamicSmemBytes = static_cast<std::size_t>(smem);
    config.stream = s;
    config.attrs = &early;
    config.numAttrs = ahead == RingAhead::ended ? 0 : 1;
    return cudaLaunchKernelEx(&config, kernel, jobs, count, ahead == RingAhead::any);
}

template <int HB, int W, int V, RingLayout LAYOUT, class In, class Out>
int rlaunch_typed(const StreamJob *jobs, int count, int blocks, RingAhead ahead, cudaStream_t s) {
    constexpr int smem = 1024 + 3 * RingRecord<HB, W>::CHUNK * 4
        + kRingThreads / 32 * (kRingBuffers * RingFeeder<In, V, W, LAYOUT>::BUFFER
                               + (LAYOUT == RingLayout::rows ? V * 4096 : 0));
    auto kernel = tring_kernel<HB, W, V, LAYOUT, In, Out>;
    static SmemLimit limit;
    if (const cudaError_t e = limit.ensure(kernel, smem); e != cudaSuccess) return static_cast<int>(e);
    return static_cast<int>(ring_launch(kernel, jobs, count, blocks, smem, ahead, s));
}

template <int HB, int W, int V>
int rlaunch(const StreamJob *jobs, int count, int blocks, dev::Sample in, dev::Sample out, RingLayout layout,
            RingAhead ahead, void *stream) {
    using dev::Sample;
    using std::uint16_t, std::uint8_t;
    using L = RingLayout;
    const auto s = static_cast<cudaStream_t>(stream);
    if (in == Sample::f32 && out == Sample::f32) {
        switch (layout) {
        case L::plain: return rlaunch_typed<HB, W, V, L::plain, float, float>(jobs, count, blocks, ahead, s);
        case L::tiled: return rlaunch_typed<HB, W, V, L::tiled, float, float>(jobs, count, blocks, ahead, s);
        case L::rows: return rlaunch_typed<HB, W, V, L::rows, float, float>(jobs, count, blocks, ahead, s);
        case L::columns: return rlaunch_typed<HB, W, V, L::columns, float, float>(jobs, count, blocks, ahead, s);
        }
    }
    if (out == Sample::f32 && layout == L::tiled) {
        if (in == Sample::u16) return rlaunch_typed<HB, W, V, L::tiled, uint16_t, float>(jobs, count, blocks, ahead, s);
        if (in == Sample::u8) return rlaunch_typed<HB, W, V, L::tiled, uint8_t, float>(jobs, count, blocks, ahead, s);
    }
    if (out == Sample::f32 && layout == L::plain) {
        if (in == Sample::u16) return rlaunch_typed<HB, W, V, L::plain, uint16_t, float>(jobs, count, blocks, ahead, s);
        if (in == Sample::u8) return rlaunch_typed<HB, W, V, L::plain, uint8_t, float>(jobs, count, blocks, ahead, s);
    }
    if (in == Sample::f32 && layout == L::plain) {
        if (out == Sample::u16) return rlaunch_typed<HB, W, V, L::plain, float, uint16_t>(jobs, count, blocks, ahead, s);
        if (out == Sample::u8) return rlaunch_typed<HB, W, V, L::plain, float, uint8_t>(jobs, count, blocks, ahead, s);
    }
    return static_cast<int>(cudaErrorInvalidValue);
}

} // namespace
} // namespace dsmvc_gb
