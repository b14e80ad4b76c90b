// Kernels of the network itself (included by mlp.cu after the tcgen05 helpers).
//
//  k_net      the whole forward pass of 128 points in one CTA and, for training,
//             the backward pass down to the first layer's pre-activations;
//  k_wgrad    weight and bias gradients of all layers, per 256 batch rows;
//  k_reduce   their sum over the batch and the Adam update.
//
// A layer is only 128 x 256 x 256 per CTA: 1.1 us of tensor-core time at the
// nominal rate, but 32768 SiLUs (an exponential and an IEEE division each, some
// 23 instructions) of 3.5 us on the SM's four schedulers, which bound the chain.
// A layer per launch spent 33 us on it -- four epilogue warps a CTA, and the
// activations out to global memory and back -- and features and output layer, one
// thread a row, 38 and 46 us more. So here sixteen warps share the epilogue, the
// activations stay in shared memory as the next layer's operand, and an epilogue
// hands them over 64 columns at a time so that the next layer's MMAs run under it.
// The loops over those chunks are not unrolled: 4 x 16 unrolled SiLUs a layer missed
// the instruction cache (24000 cycles instead of 11000 a backward layer).
//
// Measured, before -> now: training step of 16384 points, device 620 -> 112 us
// (k_net 67, k_wgrad 30, k_reduce 15), call 650 -> 150 to 163 us; forward of 19200 points
// (150 CTAs: two waves of 32 us) 409 -> 88 us. Every sum keeps the order of the
// layer-by-layer kernels it replaces, so the parameters are the same bits.
#pragma once

namespace {

constexpr int kWidth = 256;
constexpr int kFeat = 128;  // Fourier features, padded
constexpr int kFreq = 15;
constexpr int kIn = 4, kOut = 4;
constexpr int kHidden = 5;       // layers with SiLU
constexpr int kSplitRows = 256;  // batch rows per partial sum of the weight gradients
constexpr int kSplitsMax = 64;   // partial sums held at a time (1.2 MB each)

constexpr int net_din(int l) { return l == 0 ? kFeat : kWidth; }

// Offsets of the parameters (W_l row-major [out][in], then b_l) and of the BF16
// copies of W_0..W_4. All are multiples of 4.
struct NetLayout {
    int offW[kHidden + 1], offb[kHidden + 1], offWbf[kHidden];
    int nparam, nwbf;
};
NetLayout net_layout() {
    NetLayout n{};
    for (int l = 0; l <= kHidden; ++l) {
        const int out = l < kHidden ? kWidth : kOut;
        n.offW[l] = n.nparam;
        n.offb[l] = n.nparam + out * net_din(l);
        n.nparam = n.offb[l] + out;
        if (l < kHidden) {
            n.offWbf[l] = n.nwbf;
            n.nwbf += out * net_din(l);
        }
    }
    return n;
}

// Boxes of 64 x 64 of the BF16 matrices: weights [out][in], and per batch row the
// features, the activations of each layer, the pre-activations of all but the
// last hidden one, and their gradients.
struct NetMaps {
    CUtensorMap w[kHidden], f, h[kHidden], z[kHidden - 1], dz[kHidden];
    CUtensorMap part[kHidden];  // the partial sums of dW_l, [split][out][in] FP32, boxes of 32 x 32 x 1
};

struct NetArgs {
    NetLayout net;
    const float *p;      // parameters
    const float *x, *t;  // [B][4] inputs and (training) targets
    float *y, *dy;       // [B][4] outputs, or (training) loss gradient
    float *loss_part;    // per CTA, sum of (y - t)^2
    int B;
    int *err;
    unsigned wait_polls;  // bound of every wait but the final ones (kWaitLimit; 0: each gives up at once)
};

constexpr int kEpiWarps = 16, kNetThreads = 32 * (kEpiWarps + 2);
constexpr int kWStages = 3;                     // weight chunks in flight
constexpr uint32_t kBoxBytes = 64 * 64 * 2;     // one TMA box
constexpr uint32_t kActChunk = 2 * kBoxBytes;   // 64 columns of 128 rows
constexpr uint32_t kWeightChunk = 4 * kBoxBytes;  // 64 k of 256 outputs
constexpr uint32_t kActBytes = 4 * kActChunk;

// operand (h), pre-activations (training), weight stages, 1 KB to align them
template <bool TRAIN>
constexpr size_t net_smem() {
    return kActBytes * (TRAIN ? 2 : 1) + kWStages * kWeightChunk + 1024;
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// mbar_wait of a whole warp, polled in step: lanes that left a loop of their own one
// by one would stay apart for what follows.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t *bar, unsigned phase, unsigned limit) {
    for (unsigned i = 0; i < limit; ++i)
        if (__all_sync(0xffffffffu, mbar_wait(bar, phase, 1))) return true;
    return false;
}
__device__ __forceinline__ void tma_store(const CUtensorMap *map, int x, int y, const void *src) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(x), "r"(y), "r"(smem_u32(src))
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// Barrier of the warps 0-15; true if all passed true (so that a wait that ran out in one ends all).
__device__ __forceinline__ bool epi_sync(bool ok) {
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.and.pred q, 1, %2, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(all)
        : "r"((uint32_t)ok), "n"(32 * kEpiWarps)
        : "memory");
    return all != 0;
}

// N SiLUs z / (1 + e^-z) (or, DZ, factors silu'(z)) of a thread, in place. While no
// |z| of the warp reaches 87 the quotients are straight-line code with the bits of
// `/`: the compiler's own carries a branch each, which kept the N of them from
// overlapping (half the issue slots idle, 25 instead of 18 instructions).
template <bool DZ, class Div>
__device__ __forceinline__ float activation(float x, Div div) {
    const float b = 1.0f + expf(-x);
    if (!DZ) return div(x, b);
    const float s = div(1.0f, b);
    return s * (1.0f + x * (1.0f - s));
}
template <bool DZ>
__device__ __noinline__ float activation_any(float x) {
    return activation<DZ>(x, [](float a, float b) { return a / b; });
}
template <bool DZ, int N>
__device__ __forceinline__ void activate(float (&z)[N]) {
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) m = fmaxf(m, fabsf(z[i]));
    if (__all_sync(0xffffffffu, m < 87.0f)) {
#pragma unroll
        for (int i = 0; i < N; ++i) z[i] = activation<DZ>(z[i], [](float a, float b) { return psst::rn_div(a, b); });
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) z[i] = activation_any<DZ>(z[i]);
    }
}

// 16-byte unit u (8 columns) of a row in a 64-column chunk, 128-byte swizzle
__device__ __forceinline__ uint4 *act_unit(unsigned char *chunk, int row, int u) {
    return reinterpret_cast<uint4 *>(chunk + row * 128 + ((u ^ (row & 7)) << 4));
}
__device__ __forceinline__ uint4 pack8(const float *v) {
    return make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
}
__device__ __forceinline__ void unpack8(const uint4 &q, float *v) {
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v[2 * i] = __uint_as_float(w[i] << 16);
        v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}

// One CTA, 128 points. Warps 0-15 form the operands (warp w: rows 32 (w % 4)..,
// its TMEM lanes, and columns 16 (w / 4).. of each 64-column chunk), one thread
// of warp 16 issues MMAs and activation copies, one of warp 17 streams the
// weights. Steps, each "operand chunk c complete -> its MMAs": features -> layer
// 0, ..., layer 3 -> layer 4; for training then dZ_4 -> dZ_3, ..., dZ_1 -> dZ_0.
// Two accumulators alternate: the MMAs of a step start while the epilogue that
// forms their operand still reads the other.
// Barriers: hready[c], operand chunk c written (a warp's arrival each); accfull,
// all MMAs of the step done and the copies out of the operand buffers read
// (a commit and an arrival); wfull / wempty per weight stage; zfull[c],
// pre-activation chunk c loaded.
// A wait that runs out ends its role; the others' waits then run out too, and the
// CTA leaves with *err. Whatever the others do, each issuing thread sees its own MMAs
// and copies finish before the CTA's last barrier: a role that gave up no longer
// waits for them, and none may be in flight when the CTA gives its memory back.
template <bool TRAIN>
__global__ void __launch_bounds__(kNetThreads, 1) k_net(const __grid_constant__ NetMaps maps,
                                                        const __grid_constant__ NetArgs a) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char *hbuf = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    unsigned char *zbuf = hbuf + kActBytes;  // training only
    unsigned char *wbuf = hbuf + kActBytes * (TRAIN ? 2 : 1);
    __shared__ __align__(8) uint64_t wfull[kWStages], wempty[kWStages], hready[4], zfull[4], accfull;
    __shared__ uint32_t tmem_base;
    __shared__ float red[kEpiWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = blockIdx.x * kTileM;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 0) {
        for (int b = 0; b < kWStages; ++b) {
            mbar_init(&wfull[b], 1);
            mbar_init(&wempty[b], 1);
        }
        for (int c = 0; c < 4; ++c) {
            mbar_init(&hready[c], kEpiWarps);
            mbar_init(&zfull[c], 1);
        }
        mbar_init(&accfull, 2);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kEpiWarps && lane < (TRAIN ? (int)(offsetof(NetMaps, part) / sizeof(CUtensorMap)) : kHidden))
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.w[0] + lane)) : "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;
    constexpr int kSteps = TRAIN ? 2 * kHidden - 1 : kHidden;  // contractions: forward 0..4, backward 4..1
    bool ok = true;

    if (warp == kEpiWarps + 1) {
        if (lane == 0) {  // weights, in the order of use
            int n = 0;
            for (int s = 0; s < kSteps && ok; ++s) {
                const bool back = s >= kHidden;
                const int l = back ? 2 * kHidden - 1 - s : s, nch = s == 0 ? 2 : 4;
                for (int c = 0; c < nch; ++c, ++n) {
                    const int b = n % kWStages, use = n / kWStages;
                    if (use > 0 && !(ok = mbar_wait(&wempty[b], (unsigned)(use - 1) & 1u, a.wait_polls))) break;
                    mbar_expect_tx(&wfull[b], kWeightChunk);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        tma_load(wbuf + b * kWeightChunk + j * kBoxBytes, &maps.w[l], 64 * (back ? j : c),
                                 64 * (back ? c : j), &wfull[b]);
                }
            }
            for (int i = max(0, n - kWStages); i < n; ++i)  // the last copies land
                mbar_wait(&wfull[i % kWStages], (unsigned)(i / kWStages) & 1u);
        }
    } else if (warp == kEpiWarps) {
        if (lane == 0) {  // MMAs and activation copies
            int n = 0, nz = 0;
            unsigned hph = 0;  // bit c: phase of hready[c]
            auto wait_h = [&](int c) {
                const bool r = mbar_wait(&hready[c], (hph >> c) & 1u, a.wait_polls);
                hph ^= 1u << c;
                return r;
            };
            auto store = [&](const CUtensorMap *m, const unsigned char *buf, int c) {
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    if (row0 + 64 * j < a.B)
                        tma_store(m, 64 * c, row0 + 64 * j, buf + c * kActChunk + j * kBoxBytes);
            };
            for (int s = 0; s < kSteps && ok; ++s) {
                const bool back = s >= kHidden;
                const int l = back ? 2 * kHidden - 1 - s : s, nch = s == 0 ? 2 : 4;
                if (TRAIN && s == kHidden) {
                    // the last activations leave, and every pre-activation has arrived in memory, before
                    // dZ_4 takes the operand buffer and the pre-activations are read back
                    for (int c = 0; c < 4 && ok; ++c)
                        if ((ok = wait_h(c))) store(&maps.h[kHidden - 1], hbuf, c);
                    if (!ok) break;
                    bulk_commit();
                    bulk_wait();
                    asm volatile("fence.proxy.async;" ::: "memory");
                    mbar_arrive(&accfull);
                    mbar_arrive(&accfull);
                }
                const uint32_t acc = tmem + (uint32_t)(s & 1) * kWidth;
                for (int c = 0; c < nch; ++c, ++n) {
                    const int b = n % kWStages;
                    if (!(ok = wait_h(c))) break;
                    if (TRAIN) {
                        if (back) {
                            store(&maps.dz[l], hbuf, c);
                            mbar_expect_tx(&zfull[c], kActChunk);
#pragma unroll
                            for (int j = 0; j < 2; ++j)
                                tma_load(zbuf + c * kActChunk + j * kBoxBytes, &maps.z[l - 1], 64 * c, row0 + 64 * j,
                                         &zfull[c]);
                            ++nz;
                        } else {
                            store(s == 0 ? &maps.f : &maps.h[s - 1], hbuf, c);
                            if (s > 0) store(&maps.z[s - 1], zbuf, c);
                        }
                        bulk_commit();
                    }
                    if (!(ok = mbar_wait(&wfull[b], (unsigned)(n / kWStages) & 1u, a.wait_polls))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t sa = smem_u32(hbuf + c * kActChunk), sb = smem_u32(wbuf + b * kWeightChunk);
#pragma unroll
                    for (int q = 0; q < kChunkK / 16; ++q) {
                        const uint64_t da = umma_desc_sw128(sa + q * 32, 16);
                        if (back)  // W_l as stored is [k][n]: MN-major
                            umma_bf16<kWidth, false, true>(acc, da, umma_desc_sw128(sb + q * 2048, kBoxBytes),
                                                           (c > 0 || q > 0) ? 1u : 0u);
                        else
                            umma_bf16<kWidth>(acc, da, umma_desc_sw128(sb + q * 32, 16), (c > 0 || q > 0) ? 1u : 0u);
                    }
                    umma_commit(&wempty[b]);
                }
                if (!ok) break;
                umma_commit(&accfull);
                bulk_wait_read();
                mbar_arrive(&accfull);
            }
            if (TRAIN) {
                for (int c = 0; c < 4 && ok; ++c)
                    if ((ok = wait_h(c))) store(&maps.dz[0], hbuf, c);
                bulk_commit();
                bulk_wait();
            }
            // the last MMAs and copies finish
            for (int i = max(0, n - kWStages); i < n; ++i) mbar_wait(&wempty[i % kWStages], (unsigned)(i / kWStages) & 1u);
            for (int i = max(0, nz - 4); i < nz; ++i) mbar_wait(&zfull[i & 3], (unsigned)(i >> 2) & 1u);
            bulk_commit();
            bulk_wait();
        }
    } else {
        const int row = 32 * (warp & 3) + lane, grow = row0 + row, grp = warp >> 2;
        const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
        const bool in = grow < a.B;
        unsigned aph = 0, zph = 0;
        auto wait_acc = [&] {
            const bool r = mbar_wait_warp(&accfull, aph, a.wait_polls);
            aph ^= 1u;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            return r;
        };
        auto hand_over = [&](int c) {  // this warp's part of operand chunk c is written
            proxy_fence();
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&hready[c]);
        };
        {  // Fourier features of input `grp`: v, then sin and cos of 2^j pi v
            auto put = [&](int col, float f) {
                *reinterpret_cast<bf16 *>(reinterpret_cast<unsigned char *>(
                                              act_unit(hbuf + (col >> 6) * kActChunk, row, (col >> 3) & 7)) +
                                          (col & 7) * 2) = __float2bfloat16(f);
            };
            const float v = in ? a.x[(int64_t)grow * kIn + grp] : 0.0f;
            int q = grp * (2 * kFreq + 1);
            put(q++, v);
            float w = 3.14159265358979f;
            for (int j = 0; j < kFreq; ++j, w *= 2.0f) {
                float s, c;
                sincosf(w * v, &s, &c);
                put(q++, s);
                put(q++, c);
            }
            if (grp == kIn - 1)
                for (; q < kFeat; ++q) put(q, 0.0f);
            hand_over(0);
            hand_over(1);
        }
        for (int l = 0; l < kHidden && ok; ++l) {  // activations of layer l
            const float *bias = a.p + a.net.offb[l] + 16 * grp;
            const uint32_t acc = tmem + lanes + (uint32_t)(l & 1) * kWidth + 16 * grp;
            float4 b[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = __ldg(reinterpret_cast<const float4 *>(bias) + j);
            if (!(ok = wait_acc())) break;
            uint32_t r[16];
            tmem_ld16(acc, r);
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                tmem_wait(r);
                float v[16];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    v[4 * j] = __uint_as_float(r[4 * j]) + b[j].x;
                    v[4 * j + 1] = __uint_as_float(r[4 * j + 1]) + b[j].y;
                    v[4 * j + 2] = __uint_as_float(r[4 * j + 2]) + b[j].z;
                    v[4 * j + 3] = __uint_as_float(r[4 * j + 3]) + b[j].w;
                }
                if (c < 3) {
                    tmem_ld16(acc + 64 * (c + 1), r);
#pragma unroll
                    for (int j = 0; j < 4; ++j) b[j] = __ldg(reinterpret_cast<const float4 *>(bias + 64 * (c + 1)) + j);
                }
                if (TRAIN)
#pragma unroll
                    for (int u = 0; u < 2; ++u) *act_unit(zbuf + c * kActChunk, row, 2 * grp + u) = pack8(v + 8 * u);
                activate<false>(v);
#pragma unroll
                for (int u = 0; u < 2; ++u) *act_unit(hbuf + c * kActChunk, row, 2 * grp + u) = pack8(v + 8 * u);
                hand_over(c);
            }
        }
        if ((ok = epi_sync(ok))) {
            // output layer on the CUDA cores: a thread per point and output
            const float *W6 = a.p + a.net.offW[kHidden];
            float y = a.p[a.net.offb[kHidden] + grp], l = 0.0f;
#pragma unroll 8
            for (int u = 0; u < kWidth / 8; ++u) {
                float hv[8];
                unpack8(*act_unit(hbuf + (u >> 3) * kActChunk, row, u & 7), hv);
                const float4 w0 = __ldg(reinterpret_cast<const float4 *>(W6 + grp * kWidth) + 2 * u),
                             w1 = __ldg(reinterpret_cast<const float4 *>(W6 + grp * kWidth) + 2 * u + 1);
                const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
                for (int j = 0; j < 8; ++j) y += w[j] * hv[j];
            }
            const int64_t o = (int64_t)grow * kOut + grp;
            if (in) {
                if (!TRAIN) {
                    a.y[o] = y;
                } else {
                    const float d = y - a.t[o];
                    l = d * d;
                    a.dy[o] = 2.0f * d / (float)(kOut * a.B);
                }
            }
            if (TRAIN) {
                for (int s = 16; s > 0; s >>= 1) l += __shfl_down_sync(0xffffffffu, l, s);
                if (lane == 0) red[warp] = l;
                epi_sync(true);
                if (threadIdx.x == 0) {
                    float s = 0.0f;
                    for (int w = 0; w < kEpiWarps; ++w) s += red[w];
                    a.loss_part[blockIdx.x] = s;
                }
                // dZ_4 = (dy W6) silu'(z), z still in its buffer
                float dy[kOut] = {};
                if (in) {
                    const float4 d = *reinterpret_cast<const float4 *>(a.dy + (int64_t)grow * kOut);
                    dy[0] = d.x, dy[1] = d.y, dy[2] = d.z, dy[3] = d.w;
                }
                if ((ok = wait_acc())) {
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            float z[8], s[8] = {};
                            unpack8(*act_unit(zbuf + c * kActChunk, row, 2 * grp + u), z);
                            const int j0 = 64 * c + 16 * grp + 8 * u;
#pragma unroll
                            for (int k = 0; k < kOut; ++k) {
                                const float4 w0 = __ldg(reinterpret_cast<const float4 *>(W6 + k * kWidth + j0)),
                                             w1 = __ldg(reinterpret_cast<const float4 *>(W6 + k * kWidth + j0) + 1);
                                const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
                                for (int j = 0; j < 8; ++j) s[j] += dy[k] * w[j];
                            }
                            activate<true>(z);
#pragma unroll
                            for (int j = 0; j < 8; ++j) s[j] *= z[j];
                            *act_unit(hbuf + c * kActChunk, row, 2 * grp + u) = pack8(s);
                        }
                        hand_over(c);
                    }
                }
                for (int s = kHidden; s < kSteps && ok; ++s) {  // dZ_{l-1} = (dZ_l W_l) silu'(z_{l-1})
                    const uint32_t acc = tmem + lanes + (uint32_t)(s & 1) * kWidth + 16 * grp;
                    // the factors of a chunk are formed ahead of its product: the first under the MMAs
                    float v[16];
                    auto factors = [&](int c) {
                        if (!mbar_wait_warp(&zfull[c], zph, a.wait_polls)) return false;
#pragma unroll
                        for (int u = 0; u < 2; ++u)
                            unpack8(*act_unit(zbuf + c * kActChunk, row, 2 * grp + u), v + 8 * u);
                        activate<true>(v);
                        return true;
                    };
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        if (!(ok = factors(c))) break;
                        if (c == 0 && !(ok = wait_acc())) break;
                        uint32_t r[16];
                        tmem_ld16(acc + 64 * c, r);
                        tmem_wait(r);
#pragma unroll
                        for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]) * v[i];
#pragma unroll
                        for (int u = 0; u < 2; ++u)
                            *act_unit(hbuf + c * kActChunk, row, 2 * grp + u) = pack8(v + 8 * u);
                        hand_over(c);
                    }
                    zph ^= 1u;
                }
            }
        }
    }
    if (!ok) atomicExch(a.err, MLP_ERR_TIMEOUT);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

// Weight and bias gradients, partial sums of 256 batch rows each in
// part[split][parameter]. A split has 11 units: the output layer, and 128 rows of
// dW_l = dZ_l^T . H_{l-1} and db_l for each hidden layer. What bounds it is moving
// the operands (192 KB a unit for 0.6 us of MMAs) in and the partial sums (128 KB)
// out, so CTAs are persistent, one an SM, and overlap everything: one thread streams
// chunks of 64 batch rows (as stored: both operands MN-major) through four stages,
// across units; one issues MMAs into two accumulators in turn; four warps sum the
// biases and the output layer from the same stages, row by row in order; eight
// warps write finished accumulators, by TMA in 32 x 32 blocks. (A CTA per unit, two
// an SM: 41 us for 16384 rows.)
constexpr int kWgradUnits = 1 + 2 * kHidden;
constexpr int kWgradEpi = 8, kWgradSum = 4, kWgradThreads = 32 * (kWgradEpi + kWgradSum + 2);
constexpr int kWgradStages = 4;
constexpr uint32_t kWgradStage = kActChunk + kWeightChunk;  // 64 batch rows: 128 columns of dZ, up to 256 of H
constexpr size_t kWgradSmem = kWgradStages * kWgradStage + kWgradEpi * kEpiWarpBytes + 1024;

struct WgradArgs {
    NetLayout net;
    const float *dy;
    float *part;
    int B, split0, units;
    int *err;
    unsigned wait_polls;  // as in NetArgs
};

__global__ void __launch_bounds__(kWgradThreads, 1) k_wgrad(const __grid_constant__ NetMaps maps,
                                                            const __grid_constant__ WgradArgs a) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    __shared__ __align__(8) uint64_t full[kWgradStages], empty[kWgradStages], tfull[2], tempty[2], drained;
    __shared__ uint32_t tmem_base;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 0) {
        for (int b = 0; b < kWgradStages; ++b) {
            mbar_init(&full[b], 1);
            mbar_init(&empty[b], 1 + kWgradSum);  // the MMAs' commit and the summing warps
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], kWgradEpi);
        }
        mbar_init(&drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;
    bool ok = true;
    struct Unit {
        int split, l, m0, b0, rows, nchunks, din;
    };
    auto decode = [&](int u) {
        Unit t;
        const int k = u % kWgradUnits - 1;
        t.split = u / kWgradUnits;
        t.l = k < 0 ? kHidden : k >> 1;
        t.m0 = (k & 1) * kTileM;
        t.b0 = (a.split0 + t.split) * kSplitRows;
        t.rows = min(kSplitRows, a.B - t.b0);
        t.nchunks = (t.rows + 63) / 64;
        t.din = t.l == 0 ? kFeat : kWidth;
        return t;
    };
    auto full_of = [&](int n) { return &full[n % kWgradStages]; };
    auto phase_of = [&](int n) { return (unsigned)(n / kWgradStages) & 1u; };

    if (warp == kWgradEpi + kWgradSum) {
        if (lane == 0) {  // loads
            int n = 0;
            for (int u = blockIdx.x; u < a.units && ok; u += gridDim.x) {
                const Unit t = decode(u);
                const CUtensorMap *mb = t.l == 0 ? &maps.f : &maps.h[t.l - 1];
                for (int c = 0; c < t.nchunks; ++c, ++n) {
                    const int b = n % kWgradStages, row = t.b0 + 64 * c;
                    if (n >= kWgradStages && !(ok = mbar_wait(&empty[b], phase_of(n) ^ 1u, a.wait_polls))) break;
                    unsigned char *sa = smem + b * kWgradStage, *sb = sa + kActChunk;
                    const uint32_t bb = (uint32_t)(t.din / 64) * kBoxBytes;
                    if (t.l == kHidden) {
                        const uint32_t bytes = 16u * (uint32_t)min(64, t.rows - 64 * c);
                        mbar_expect_tx(&full[b], bb + bytes);
                        asm volatile(
                            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                smem_u32(sa)),
                            "l"(a.dy + (int64_t)row * kOut), "r"(bytes), "r"(smem_u32(&full[b]))
                            : "memory");
                    } else {
                        mbar_expect_tx(&full[b], bb + kActChunk);
                        for (int j = 0; j < 2; ++j) tma_load(sa + j * kBoxBytes, &maps.dz[t.l], t.m0 + 64 * j, row, &full[b]);
                    }
                    for (int j = 0; j < t.din / 64; ++j) tma_load(sb + j * kBoxBytes, mb, 64 * j, row, &full[b]);
                }
            }
            for (int i = max(0, n - kWgradStages); i < n; ++i) mbar_wait(full_of(i), phase_of(i));  // the last copies land
        }
    } else if (warp == kWgradEpi + kWgradSum + 1) {
        if (lane == 0) {  // MMAs
            int n = 0, k = 0;
            for (int u = blockIdx.x; u < a.units && ok; u += gridDim.x) {
                const Unit t = decode(u);
                const uint32_t acc = tmem + (uint32_t)(k & 1) * kWidth;
                if (t.l < kHidden && k >= 2 && !(ok = mbar_wait(&tempty[k & 1], (unsigned)((k >> 1) - 1) & 1u, a.wait_polls))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int c = 0; c < t.nchunks; ++c, ++n) {
                    const int b = n % kWgradStages;
                    if (!(ok = mbar_wait(&full[b], phase_of(n), a.wait_polls))) break;
                    if (t.l == kHidden) {
                        mbar_arrive(&empty[b]);
                        continue;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t sa = smem_u32(smem + b * kWgradStage), sb = sa + kActChunk;
#pragma unroll
                    for (int q = 0; q < kChunkK / 16; ++q) {
                        const uint64_t da = umma_desc_sw128(sa + q * 2048, kBoxBytes),
                                       db = umma_desc_sw128(sb + q * 2048, kBoxBytes);
                        const uint32_t more = (c > 0 || q > 0) ? 1u : 0u;
                        if (t.l == 0)
                            umma_bf16<kFeat, true, true>(acc, da, db, more);
                        else
                            umma_bf16<kWidth, true, true>(acc, da, db, more);
                    }
                    umma_commit(&empty[b]);
                }
                if (!ok) break;
                if (t.l < kHidden) umma_commit(&tfull[k++ & 1]);
            }
            umma_commit(&drained);
            ok = mbar_wait(&drained, 0) && ok;
        }
    } else if (warp >= kWgradEpi) {
        // thread j: db_l[m0 + j]; for the output layer dW[.][2j], dW[.][2j + 1]
        const int j = threadIdx.x - 32 * kWgradEpi;
        int n = 0;
        for (int u = blockIdx.x; u < a.units && ok; u += gridDim.x) {
            const Unit t = decode(u);
            float *part = a.part + (int64_t)t.split * a.net.nparam;
            float s = 0.0f, s0[kOut] = {}, s1[kOut] = {}, sb[kOut] = {};
            for (int c = 0; c < t.nchunks; ++c, ++n) {
                const int b = n % kWgradStages;
                if (!(ok = mbar_wait_warp(&full[b], phase_of(n), a.wait_polls))) break;
                const unsigned char *sa = smem + b * kWgradStage;
                if (t.l < kHidden) {
                    const unsigned char *box = sa + (j >> 6) * kBoxBytes + (j & 7) * 2;
                    const int unit = (j >> 3) & 7;
#pragma unroll 16
                    for (int r = 0; r < 64; ++r)  // rows past the batch are zeros
                        s += __bfloat162float(*reinterpret_cast<const bf16 *>(box + r * 128 + ((unit ^ (r & 7)) << 4)));
                } else {
                    const unsigned char *box = sa + kActChunk + (j >> 5) * kBoxBytes + (j & 3) * 4;
                    const int unit = (j >> 2) & 7, rows = min(64, t.rows - 64 * c);
#pragma unroll 8
                    for (int r = 0; r < rows; ++r) {
                        const uint32_t w = *reinterpret_cast<const uint32_t *>(box + r * 128 + ((unit ^ (r & 7)) << 4));
                        const float h0 = __uint_as_float(w << 16), h1 = __uint_as_float(w & 0xffff0000u);
                        const float4 d = reinterpret_cast<const float4 *>(sa)[r];
                        s0[0] += d.x * h0, s0[1] += d.y * h0, s0[2] += d.z * h0, s0[3] += d.w * h0;
                        s1[0] += d.x * h1, s1[1] += d.y * h1, s1[2] += d.z * h1, s1[3] += d.w * h1;
                        sb[0] += d.x, sb[1] += d.y, sb[2] += d.z, sb[3] += d.w;
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[b]);
            }
            if (!ok) break;
            if (t.l < kHidden) {
                part[a.net.offb[t.l] + t.m0 + j] = s;
            } else {
#pragma unroll
                for (int o = 0; o < kOut; ++o) {
                    *reinterpret_cast<float2 *>(part + a.net.offW[kHidden] + o * kWidth + 2 * j) = make_float2(s0[o], s1[o]);
                    if (j == 0) part[a.net.offb[kHidden] + o] = sb[o];
                }
            }
        }
    } else {
        // rows 32 (warp % 4).., half of the columns
        const int r0 = 32 * (warp & 3);
        unsigned char *tile = smem + kWgradStages * kWgradStage + warp * kEpiWarpBytes;
        int k = 0;
        for (int u = blockIdx.x; u < a.units; u += gridDim.x) {
            const Unit t = decode(u);
            if (t.l == kHidden) continue;
            const uint32_t acc = tmem + ((uint32_t)r0 << 16) + (uint32_t)(k & 1) * kWidth;
            if (!(ok = mbar_wait_warp(&tfull[k & 1], (unsigned)(k >> 1) & 1u, a.wait_polls))) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int half = t.din / 2;
            for (int c0 = 0; c0 < half; c0 += 32) {
                const int col = (warp >> 2) * half + c0;
                float v[32];
                tmem_ld32(acc + (uint32_t)col, v);
                if (lane == 0) bulk_wait_read();
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    *tile32(tile, lane, j) = make_uint4(__float_as_uint(v[4 * j]), __float_as_uint(v[4 * j + 1]),
                                                        __float_as_uint(v[4 * j + 2]), __float_as_uint(v[4 * j + 3]));
                proxy_fence();
                __syncwarp();
                if (lane == 0) {
                    asm volatile(
                        "cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(
                            reinterpret_cast<uint64_t>(&maps.part[t.l])),
                        "r"(col), "r"(t.m0 + r0), "r"(t.split), "r"(smem_u32(tile))
                        : "memory");
                    bulk_commit();
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[k & 1]);
            ++k;
        }
        if (lane == 0) bulk_wait();
    }
    if (!ok) atomicExch(a.err, MLP_ERR_TIMEOUT);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

struct AdamArgs {
    NetLayout net;
    float *p, *m, *v;
    bf16 *wbf;
    float lr, b1, b2, eps, c1, c2;
};
struct LossArgs {
    const float *part;
    int n;
    double scale;
    int *status;  // error word, loss
};

// BF16 copies of the tensor-core weights among parameters 4i..4i+3.
__device__ __forceinline__ void refresh_bf16(const NetLayout &net, int i, const float p[4], bf16 *wbf) {
#pragma unroll
    for (int l = 0; l < kHidden; ++l)
        if (i >= net.offW[l] && i < net.offb[l])
            *reinterpret_cast<uint2 *>(wbf + net.offWbf[l] + i - net.offW[l]) =
                make_uint2(pack_bf16(p[0], p[1]), pack_bf16(p[2], p[3]));
}

// Gradient = sum of the splits' partial sums in order (added to g unless first),
// four parameters a thread; then into g, or (ADAM: Kingma & Ba, 2015) into the
// FP32 master parameters. The first CTA also sums the loss. Nothing is applied
// after a wait that ran out.
template <bool ADAM>
__global__ void k_reduce(const float *part, int splits, int n4, bool first, float *g,
                         const __grid_constant__ AdamArgs a, const LossArgs loss) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.x == 0 && threadIdx.x < 32) {
        double s = 0.0;
        for (int k = threadIdx.x; k < loss.n; k += 32) s += loss.part[k];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) reinterpret_cast<float *>(loss.status)[1] = (float)(s * loss.scale);
    }
    if (i >= n4 || *loss.status) return;
    float s[4] = {};
    if (!first) {
        const float4 q = reinterpret_cast<const float4 *>(g)[i];
        s[0] = q.x, s[1] = q.y, s[2] = q.z, s[3] = q.w;
    }
#pragma unroll 16
    for (int z = 0; z < splits; ++z) {
        const float4 q = __ldcs(reinterpret_cast<const float4 *>(part) + (int64_t)z * n4 + i);
        s[0] += q.x, s[1] += q.y, s[2] += q.z, s[3] += q.w;
    }
    if (!ADAM) {
        reinterpret_cast<float4 *>(g)[i] = make_float4(s[0], s[1], s[2], s[3]);
        return;
    }
    float4 *pm = reinterpret_cast<float4 *>(a.m) + i, *pv = reinterpret_cast<float4 *>(a.v) + i,
           *pp = reinterpret_cast<float4 *>(a.p) + i;
    const float4 qm = *pm, qv = *pv, qp = *pp;
    float m[4] = {qm.x, qm.y, qm.z, qm.w}, v[4] = {qv.x, qv.y, qv.z, qv.w}, p[4] = {qp.x, qp.y, qp.z, qp.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        m[k] = fmaf(1.0f - a.b1, s[k], a.b1 * m[k]);
        v[k] = fmaf((1.0f - a.b2) * s[k], s[k], a.b2 * v[k]);
        p[k] = p[k] - a.lr * (m[k] / a.c1) / (sqrtf(v[k] / a.c2) + a.eps);
    }
    *pm = make_float4(m[0], m[1], m[2], m[3]);
    *pv = make_float4(v[0], v[1], v[2], v[3]);
    *pp = make_float4(p[0], p[1], p[2], p[3]);
    refresh_bf16(a.net, 4 * i, p, a.wbf);
}

__global__ void k_to_bf16(const float *p, NetLayout net, bf16 *wbf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (4 * i >= net.nparam) return;
    const float4 q = reinterpret_cast<const float4 *>(p)[i];
    const float v[4] = {q.x, q.y, q.z, q.w};
    refresh_bf16(net, 4 * i, v, wbf);
}

}  // namespace
