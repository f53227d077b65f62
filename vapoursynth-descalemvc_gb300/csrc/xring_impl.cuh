// Two-pass transposing kernels with the sample ring in tensor memory: the exact
// 2D passes of a Float32 descale, for plans whose factors decay too slowly for
// one chunk of warm-up and half-bandwidths up to 11.
//
// Loads, ring and records as in tring_impl.cuh; the substitution runs as two
// sweeps over the vector:
//
//  * forward sweep, first destination to last: the gather and the forward
//    substitution in the reference CUDA order, each forward value stored to a
//    Float32 plane laid out like the output (one coalesced store);
//  * backward sweep, last chunk to first: the forward values of a group of
//    destinations loaded one group ahead, the backward substitution in the
//    reference order from the exact carry of the chunk after it.
//
// Nothing is approximated, so whole vectors equal the reference CUDA kernels'
// bit for bit; segments (StreamJob) start from margins.  The forward plane is
// the output itself where it is a Float32 plane (the first pass's
// intermediate, Float32 outputs), else a caller scratch plane.
//
// What bounds them: a half-bandwidth 9 result takes 36 FMA slots (two 16-tap
// gathers cannot share a packed FMA in this order) and nine 16-byte record
// loads of two shared-memory cycles each; small launches wait on one vector's
// chain.  Both lane counts spill under their caps of 128 and 168 registers: at
// half-bandwidths 9 and 11, 40-80 bytes stored and 76-136 loaded a lane at one vector,
// 100-140 and 216-280 at two, whose loops take 16 destinations at a time.  Measured on one GB300 against the kernels with ring in shared memory
// and a refill per destination: eight 4K Float32 frames to 1440p, Spline64 blur
// 1.1, 859 -> 447 us; a 1080p sweep of 189 candidates, of which 33 run these,
// 3911 -> 3084.
#pragma once

#include "tring_impl.cuh"

namespace dsmvc_gb {
namespace {

// One half of a chunk's records, forward or backward.
__device__ __forceinline__ void xstage(float *buf, const float *from, int floats, int tid) {
    for (int i = tid * 4; i < floats; i += kRingThreads * 4) tcp_async16(buf + i, from + i);
}

template <int HB, int W, int V, bool TILED, class In, class Out>
__global__ void __launch_bounds__(kRingThreads, V == 1 ? 4 : 3)
xring_kernel(const StreamJob *__restrict__ jobs, int job_count, bool late) {
    using R = RingRecord<HB, W>;
    using Feed = RingFeeder<In, V, W, RingLayout::plain>;
    constexpr int LC = kTChunk, WARPS = kRingThreads / 32, G = 8;
    constexpr int FORWARD = R::GROUPS * R::GROUP, BACKWARD = R::GROUPS * R::LOW;
    constexpr int COLUMNS = V * Feed::VC;
    static_assert(COLUMNS == 64 || COLUMNS == 128);
    extern __shared__ unsigned char ring_dynamic[];
    unsigned char *const ring_smem = ring_dynamic + (-static_cast<unsigned>(__cvta_generic_to_shared(ring_dynamic)) & 1023);
    float *bufs = reinterpret_cast<float *>(ring_smem + WARPS * kRingBuffers * Feed::BUFFER);   // 3 * FORWARD
    __shared__ unsigned long long feed_bar[WARPS][kRingBuffers];
    __shared__ unsigned tm_base;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // Jobs are assigned warps; a CTA's warps share one plan and chunk range.
    const int cta_warp = static_cast<int>(blockIdx.x) * WARPS;
    const StreamJob &job = jobs[find_tjob(jobs, job_count, cta_warp + warp)];
    const StreamJob &lead = jobs[find_tjob(jobs, job_count, cta_warp)];
    const dev::StreamPlanView p = lead.plan;
    const int n = p.destination_size;
    const int chunks = (n + LC - 1) / LC;
    // Chunks stored: [ca, cb); a segment (chunk_end > 0) sweeps forward over
    // [fc0, fce] from a zero history and backward from a zero carry after
    // fce, `margin` chunks beyond its range on either side (within the
    // vector), with its forward values in its own region from chunk fc0 on.
    const bool segment = lead.chunk_end > 0;
    const int ca = lead.chunk_begin;
    const int cb = segment ? lead.chunk_end : chunks;
    const int fc0 = segment ? max(ca - lead.margin, 0) : 0;
    const int fce = segment ? min(cb + lead.margin, chunks) - 1 : chunks - 1;

    xstage(bufs + (fc0 % 3) * FORWARD, p.forward + static_cast<std::int64_t>(fc0) * FORWARD, FORWARD, tid);
    tcp_commit();
    if (fc0 + 1 <= fce)
        xstage(bufs + ((fc0 + 1) % 3) * FORWARD, p.forward + static_cast<std::int64_t>(fc0 + 1) * FORWARD, FORWARD, tid);
    tcp_commit();
    if (!late) ring_allocate<COLUMNS>(&tm_base, warp);
    if (lane < kRingBuffers) {
        const unsigned mb = static_cast<unsigned>(__cvta_generic_to_shared(&feed_bar[warp][lane]));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" :: "r"(mb), "r"(ring_arrivals<RingLayout::plain>(job, lead)) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    ring_allocated();

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
    if (!idle) feed.start(fc0 > 0 ? lead.first_sample : 0, tm + (static_cast<unsigned>(warp * 32) << 16));
    ring_launch_next();

    // Forward value of destination j at yp[a][j * y_elem].  Lanes past the
    // warp's last vector repeat it.  The tiled intermediate holds whole
    // vectors' forward values too.
    const bool y_tiled = TILED && !segment;
    const std::int64_t y_elem = y_tiled ? 32 : job.y_elem, out_elem = TILED ? 32 : job.out_elem;
    const Conversion conv = job.conv;
    float *yp[V];
    Out *out[V];
#pragma unroll
    for (int a = 0; a < V; ++a) {
        const int v = idle ? 0 : warp_first + min(lane + 32 * a, feed.vectors - 1);
        const std::int64_t in_tile = static_cast<std::int64_t>(v >> 5) * n * 32 + (v & 31);
        yp[a] = job.y + (y_tiled ? in_tile : v) - static_cast<std::int64_t>(segment ? fc0 * LC : 0) * y_elem;
        out[a] = static_cast<Out *>(job.out) + (TILED ? in_tile : v);
    }

    // ---- forward sweep ---------------------------------------------------
    float hist[V][HB];
#pragma unroll
    for (int a = 0; a < V; ++a)
#pragma unroll
        for (int d = 0; d < HB; ++d) hist[a][d] = 0.0f;
    for (int c = fc0; c <= fce; ++c) {
        tcp_wait_one();
        __syncthreads();
        if (!idle) {
            const int j0 = c * LC;
            rforward<HB, W, V, false>(hist, bufs + (c % 3) * FORWARD, feed, [&](int a, int t, const float *y) {
                float *to = yp[a] + (j0 + t) * y_elem;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (j0 + t + i < n) *to = y[i];
                    to += y_elem;
                }
            });
        }
        __syncthreads();
        if (c + 2 <= fce)
            xstage(bufs + ((c + 2) % 3) * FORWARD, p.forward + static_cast<std::int64_t>(c + 2) * FORWARD, FORWARD, tid);
        tcp_commit();
    }

    // ---- backward sweep --------------------------------------------------
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    xstage(bufs, p.backward + static_cast<std::int64_t>(fce) * BACKWARD, BACKWARD, tid);
    tcp_commit();
    if (fce - 1 >= ca)
        xstage(bufs + BACKWARD, p.backward + static_cast<std::int64_t>(fce - 1) * BACKWARD, BACKWARD, tid);
    tcp_commit();
    float carry[V][HB], next[V][G];
    // The forward values of destinations [j, j + G): those of the vector.
    auto fetch = [&](int j) {
#pragma unroll
        for (int a = 0; a < V; ++a) {
            const float *from = yp[a] + j * y_elem;
#pragma unroll
            for (int t = 0; t < G; ++t) {
                next[a][t] = j + t < n ? *from : 0.0f;
                from += y_elem;
            }
        }
    };
#pragma unroll
    for (int a = 0; a < V; ++a)
#pragma unroll
        for (int d = 0; d < HB; ++d) carry[a][d] = 0.0f;
    if (!idle) fetch(fce * LC + LC - G);
    for (int c = fce, k = 0; c >= ca; --c, ++k) {
        const int j0 = c * LC;
        // Results to store: destinations [j0, j0 + stored).
        const int stored = c < cb ? min(LC, n - j0) : 0;
        tcp_wait_one();
        __syncthreads();
        const float *bwd = bufs + (k % 3) * BACKWARD;
        if (!idle) {
#pragma unroll 1
            for (int tg = LC - G; tg >= 0; tg -= G) {
                float x[V][G + HB];
#pragma unroll
                for (int a = 0; a < V; ++a) {
#pragma unroll
                    for (int t = 0; t < G; ++t) x[a][t] = next[a][t];
#pragma unroll
                    for (int d = 0; d < HB; ++d) x[a][G + d] = carry[a][d];
                }
                if (j0 + tg > ca * LC) fetch(j0 + tg - G);
                // Lanes that repeat a vector share its plane in place: all
                // have read the next group before one stores there.
                __syncwarp();
                float u[2][R::LOW];
                rload(u[1], bwd + (tg / 4 + 1) * R::LOW);
                rload(u[0], bwd + (tg / 4) * R::LOW);
#pragma unroll
                for (int t = G - 1; t >= 0; --t) {
#pragma unroll
                    for (int a = 0; a < V; ++a) {
                        float sum = 0.0f;
#pragma unroll
                        for (int pos = 0; pos < HB; ++pos)
                            sum = fmaf(u[t / 4][(t % 4) * HB + pos], x[a][t + (HB == 3 ? pos + 1 : HB - pos)], sum);
                        x[a][t] = x[a][t] - sum;
                    }
                }
#pragma unroll
                for (int a = 0; a < V; ++a) {
                    Out *to = out[a] + (j0 + tg) * out_elem;
#pragma unroll
                    for (int t = 0; t < G; ++t) {
                        if (tg + t < stored) *to = rout<Out>(x[a][t], conv);
                        to += out_elem;
                    }
#pragma unroll
                    for (int d = 0; d < HB; ++d) carry[a][d] = x[a][d];
                }
            }
        }
        __syncthreads();
        if (c - 2 >= ca)
            xstage(bufs + ((k + 2) % 3) * BACKWARD, p.backward + static_cast<std::int64_t>(c - 2) * BACKWARD, BACKWARD, tid);
        tcp_commit();
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    if (!idle) feed.drain();
    if (__any_sync(0xffffffffu, feed.failed) && lane == 0) atomicOr(lead.status, dev::kStatusFeedStall);
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" :: "r"(tm), "n"(COLUMNS));
}

template <int HB, int W, int V, bool TILED, class In, class Out>
int xrlaunch_typed(const StreamJob *jobs, int count, int blocks, RingAhead ahead, cudaStream_t s) {
    using R = RingRecord<HB, W>;
    constexpr int smem = 1024 + 3 * R::GROUPS * R::GROUP * 4
        + kRingThreads / 32 * kRingBuffers * RingFeeder<In, V, W, RingLayout::plain>::BUFFER;
    auto kernel = xring_kernel<HB, W, V, TILED, In, Out>;
    static SmemLimit limit;
    if (const cudaError_t e = limit.ensure(kernel, smem); e != cudaSuccess) return static_cast<int>(e);
    return static_cast<int>(ring_launch(kernel, jobs, count, blocks, smem, ahead, s));
}

template <int HB, int W, int V>
int xrlaunch(const StreamJob *jobs, int count, int blocks, dev::Sample in, dev::Sample out, bool tiled,
             RingAhead ahead, void *stream) {
    using dev::Sample;
    using std::uint16_t, std::uint8_t;
    const auto s = static_cast<cudaStream_t>(stream);
    if (out == Sample::f32) {
        if (in == Sample::f32)
            return tiled ? xrlaunch_typed<HB, W, V, true, float, float>(jobs, count, blocks, ahead, s)
                         : xrlaunch_typed<HB, W, V, false, float, float>(jobs, count, blocks, ahead, s);
        if (in == Sample::u16)
            return tiled ? xrlaunch_typed<HB, W, V, true, uint16_t, float>(jobs, count, blocks, ahead, s)
                         : xrlaunch_typed<HB, W, V, false, uint16_t, float>(jobs, count, blocks, ahead, s);
        if (in == Sample::u8)
            return tiled ? xrlaunch_typed<HB, W, V, true, uint8_t, float>(jobs, count, blocks, ahead, s)
                         : xrlaunch_typed<HB, W, V, false, uint8_t, float>(jobs, count, blocks, ahead, s);
    }
    if (in == Sample::f32 && out == Sample::u16)
        return xrlaunch_typed<HB, W, V, false, float, uint16_t>(jobs, count, blocks, ahead, s);
    if (in == Sample::f32 && out == Sample::u8)
        return xrlaunch_typed<HB, W, V, false, float, uint8_t>(jobs, count, blocks, ahead, s);
    return static_cast<int>(cudaErrorInvalidValue);
}

} // namespace
} // namespace dsmvc_gb
