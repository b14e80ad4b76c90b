// A whole psst_explicit_solve call as one persistent, cooperative launch that
// passes cell states from cell to cell instead of stopping at grid barriers.
//
// Two uses, one kernel:
//  * the sequential LocalAccTime1 (the reference evaluates it inside its update
//    loop, psstFiniteVolumeGrid.cpp:317-323, so within a stage each cell sees
//    the neighbours updated before it: a Gauss-Seidel chain), any mesh, FP64;
//  * the parallel time-step modes on small meshes, where a pass of the
//    launch-by-launch form has too few cells to fill the chip and an iteration
//    is a chain of ten launches.
//
// Operations of the call (per iteration the gradient when the scheme has one,
// then the RK stages) are numbered m; cells are grouped into items of 32 cells
// of one level (ResSched; one level in the parallel modes), four lanes a cell.
// Every CTA owns a fixed set of items and runs its (item, operation) pairs in
// the order P m + level. An operation needs, of each neighbouring cell, the
// result of operation m - 1 (or of m itself, for neighbours of a lower level
// that the reference updates first); all of these come earlier in that order,
// and all CTAs are co-resident, so the oldest unfinished pair can always run.
//
// What a neighbour needs is published in records whose every 64-bit word holds
// its own tag (Record below): the reader polls the record itself until the tags
// say that it holds the operation
// asked for. So a result costs one store and one load through L2 (541 cycles
// one way, measured between two SMs) -- no fence, no flag, no barrier. States
// are double-buffered by stage parity and gradient projections single-buffered:
// a cell overwrites a slot only after it has read, from every neighbour, a
// result that the neighbour formed after reading that slot. Gradients are
// published per face, already projected on the offset that the face needs (4 or
// 5 values instead of 8 or 15).
//
// A call is bound by the latency of one operation's instructions on one warp,
// not by memory (the meshes fit L2), and everyone waits for the slowest warp.
// So: a face a lane, each interior face's flux formed by both of its cells with
// the same arithmetic; straight-line code with selects instead of branches
// (boundary faces and all wave patterns take the same path; exact.cuh's
// divisions and square roots); sums over the faces after a transpose through
// shuffles, lane v adding component v in the reference's order, so FP64 results
// are the reference's bit for bit; static face data in one coalesced record per
// lane. One lane a cell, four faces interleaved, was measured too: 3640
// instructions an operation and twice the time.
//
// Measured (a whole call, state in to state out, launch-by-launch or one-CTA-a-level
// chain before -> now): 60 x 20 FP64, one iteration 155 -> 113 us; 120 x 40 FP64,
// 100 iterations 5.23 -> 2.00 ms; 240 x 80 FP32, 50 iterations 2.11 -> 1.45 ms;
// sequential 240 x 80 (first order, 300) 8.56 -> 4.16 ms and 120 x 40 (30) 4.16 -> 1.53
// ms. An operation of the 120 x 40 case takes some 7900 cycles; of the 8300 that a copy
// with clock64 in it took: 900 for the static data, 900 waiting for neighbours, 2400
// fluxes, 800 the sums over the faces, 1450 update and
// publication, 550 ghosts, 350 norms, 900 the loop and its barrier.
//
// Every wait is bounded: one longer than wait_ns sets the abort flag and
// ERR_TIMEOUT, and every warp leaves at its next wait of 256 attempts (data that
// arrives sooner is what it waited for). A warp that gave up forms and publishes
// nothing from what it has.
#pragma once
#include <type_traits>

#include "exact.cuh"
#include "kernels.cuh"
#include "ops.hpp"

namespace psst {

__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Published records: 64-bit words of 32 bits of data and a 32-bit tag, moved
// four at a time (one 32-byte sector per request) by relaxed vector accesses,
// each word of which is written and read whole. An FP32 value takes one word, an
// FP64 value two; a reader takes a record once every word carries the tag it
// waits for. (Words of 16 bytes read one by one cost 5 requests of 32 sectors a
// warp for a state, and the requests, not the latency, set the pace: 6800 cycles
// an exchange, measured.)
template <typename R>
constexpr int record_words(int n) {  // of n values, in whole sectors
    return (n * (int)(sizeof(R) / 4) + 3) / 4 * 4;
}
template <typename R, int N>
struct Record {
    static constexpr int W = record_words<R>(N);
    uint64_t w[W];
    __device__ __forceinline__ bool holds(uint32_t tag) const {
        bool ok = true;
#pragma unroll
        for (int i = 0; i < W; ++i) ok = ok && (uint32_t)(w[i] >> 32) == tag;
        return ok;
    }
    __device__ __forceinline__ R value(int i) const {
        if constexpr (sizeof(R) == 8)
            return __hiloint2double((int)(uint32_t)w[2 * i + 1], (int)(uint32_t)w[2 * i]);
        else
            return __uint_as_float((uint32_t)w[i]);
    }
    __device__ __forceinline__ void fetch(const uint64_t *p) {
#pragma unroll
        for (int i = 0; i < W; i += 4)
            asm volatile("ld.relaxed.gpu.global.v4.b64 {%0, %1, %2, %3}, [%4];"
                         : "=l"(w[i]), "=l"(w[i + 1]), "=l"(w[i + 2]), "=l"(w[i + 3])
                         : "l"(p + i)
                         : "memory");
    }
};
// Sector k of the record of v[0 .. N).
template <typename R, int N>
__device__ __forceinline__ void publish_sector(uint64_t *p, int k, const R *v, uint32_t tag) {
    constexpr int PER = sizeof(R) == 8 ? 2 : 4;  // values in a sector
    const uint64_t t = (uint64_t)tag << 32;
    uint64_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = t;
#pragma unroll
    for (int s = 0; s < record_words<R>(N) / 4; ++s)
        if (k == s)
#pragma unroll
            for (int i = 0; i < PER; ++i)
                if (s * PER + i < N) {
                    if constexpr (sizeof(R) == 8) {
                        w[2 * i] = t | (uint32_t)__double2loint(v[s * PER + i]);
                        w[2 * i + 1] = t | (uint32_t)__double2hiint(v[s * PER + i]);
                    } else {
                        w[i] = t | __float_as_uint(v[s * PER + i]);
                    }
                }
    asm volatile("st.relaxed.gpu.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p + 4 * k), "l"(w[0]), "l"(w[1]),
                 "l"(w[2]), "l"(w[3])
                 : "memory");
}

// sync[0] counts CTAs that have finished (monotonic over launches),
// sync[kSyncAbort] is the abort flag, each on its own 128-byte line.
constexpr int kSyncAbort = 64;
static_assert(kSyncAbort < kWfSyncWords, "sync words");

// Bounded waiting: again() is called after every unsuccessful attempt and says
// whether to try once more. The clock and the abort flag are looked at rarely
// (a failed attempt costs one load through L2), the flag by a relaxed load: an
// acquire would empty the SM's L1, which holds the static face data.
struct Waiter {
    unsigned *sync;
    int32_t *err;
    uint64_t limit_ns;
    uint64_t t0;
    unsigned spins;
    __device__ __forceinline__ bool again(int where) {
        if ((++spins & 255u) != 0u && limit_ns != 0) return true;
        const uint64_t now = global_ns();
        if (spins <= 256u) t0 = now;
        unsigned stop;
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(stop) : "l"(&sync[kSyncAbort]) : "memory");
        if (stop != 0u) return false;
        if (limit_ns == 0 || now - t0 > limit_ns) {
            atomicExch(&sync[kSyncAbort], 1u);
            flag_error(err, ERR_TIMEOUT, where);
            return false;
        }
        return true;
    }
};

// After it, lane q of each quad holds in v[j] what lane j held in v[q].
template <typename R>
__device__ __forceinline__ void quad_transpose(R v[4], int q) {
#pragma unroll
    for (int h = 0; h < 4; h += 2) {
        const R t = __shfl_xor_sync(FULL, (q & 1) ? v[h] : v[h + 1], 1);
        if (q & 1)
            v[h] = t;
        else
            v[h + 1] = t;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const R t = __shfl_xor_sync(FULL, (q & 2) ? v[h] : v[h + 2], 2);
        if (q & 2)
            v[h] = t;
        else
            v[h + 2] = t;
    }
}

template <typename R, int N>
__device__ __forceinline__ R pick(const R v[N], int i) {
    R x = v[0];
#pragma unroll
    for (int k = 1; k < N; ++k)
        if (i == k) x = v[k];
    return x;
}

// a published state: u.., p, T, rho (value i < DIM + 2 is variable i of pvar)
template <typename R, int DIM>
__device__ __forceinline__ Prim<R, DIM> from_record(const Record<R, DIM + 3> &w) {
    Prim<R, DIM> s;
#pragma unroll
    for (int k = 0; k < DIM; ++k) s.u[k] = w.value(k);
    s.p = w.value(DIM);
    s.T = w.value(DIM + 1);
    s.rho = w.value(DIM + 2);
    return s;
}

// Static data of one face of one lane's cell: the neighbours (nb across the face
// at this position of the face-loop order, -1: no such face; nb2 across the face
// at the same position of the cell's own order), the lane record of the same face
// in the cell across (kFaceLocal: a cell of the same item), flags, and the fields n, S | off (the face's reconstruction
// offset on this side), g (Green-Gauss: signed S / V, beta, in FP32 the weight of
// the cell across and signed S n / V; least squares: the weights of nb2) | n2, S2
// (of nb2's face). Kept in 16-byte pieces, piece-major
// over the lanes, so that a warp's load is one run of 512 bytes; formed once by
// k_res_build from the grid's own arrays with their arithmetic.
constexpr uint32_t kFaceSide = 1, kFaceInner = 2, kFaceLow = 4, kFaceSame = 8, kFaceValid = 16, kFaceLocal = 32;
template <typename R, int DIM>
struct FaceData {
    static constexpr int PER = 16 / (int)sizeof(R);              // fields in a piece
    static constexpr int NS = (DIM + 1 + PER - 1) / PER;         // pieces of n, S
    static constexpr int OG = (DIM + 3 + PER - 1) / PER;         // pieces of off, g
    static constexpr int OFFP = (DIM + PER - 1) / PER;           // the first of them: off
    static constexpr int PIECES = 1 + 2 * NS + OG;
    static_assert(sizeof(R) == 8 || 2 * DIM + 1 <= OG * PER, "off and the FP32 Green-Gauss coefficients");
    // pieces [A, A + N) after the ids of lane `t` of a face block, as R values
    template <int A, int N>
    static __device__ __forceinline__ void fields(const uint4 *block, int t, R *out) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const uint4 w = __ldg(block + (1 + A + i) * kWfBlock + t);
            memcpy(out + i * PER, &w, 16);
        }
    }
};

template <typename R, int DIM>
__global__ void __launch_bounds__(kWfBlock) k_res_build(DevGrid g, int rec, int grad, const int32_t *cells32,
                                                        const uint32_t *lowmask, const int32_t *mate,
                                                        const int32_t *pos, int rounds, uint4 *faces, double2 *cells) {
    using FD = FaceData<R, DIM>;
    constexpr bool EXACT = sizeof(R) == 8;
    const int item = blockIdx.x / rounds, round = blockIdx.x % rounds, t = threadIdx.x, slot = t / 4, q = t % 4;
    const int32_t c = cells32[(size_t)item * 32 + slot];
    const int j = 4 * round + q;
    int4 ids = make_int4(-1, -1, 0, 0);
    R f[(FD::PIECES - 1) * FD::PER];
#pragma unroll
    for (int i = 0; i < (FD::PIECES - 1) * FD::PER; ++i) f[i] = (R)0;
    R *ns = f, *og = f + FD::NS * FD::PER, *ns2 = og + FD::OG * FD::PER;
    const int32_t b = c >= 0 ? g.csr_ptr[c] : 0, K = c >= 0 ? g.csr_ptr[c + 1] - b : 0;
    if (j < K) {
        const FaceRec<R, DIM> *frec = reinterpret_cast<const FaceRec<R, DIM> *>(g.frec);
        const int slot2 = (int)((g.wperm[c] >> (4 * j)) & 15);
        const int32_t ent = g.csr_ent[b + j], side = ent & 1;
        const FaceRec<R, DIM> fr = frec[ent >> 1], fr2 = frec[g.csr_ent[b + slot2] >> 1];
        ids.x = g.csr_nb[b + j];
        ids.y = g.csr_nb[b + slot2];
        uint32_t bits = kFaceValid | (side ? kFaceSide : 0u) | (slot2 == j ? kFaceSame : 0u);
        if (ids.x < g.nint) {
            bits |= kFaceInner;
            const int32_t jm = mate[b + j] - g.csr_ptr[ids.x], p = pos[ids.x];
            ids.z = ((p / 32) * rounds + jm / 4) * kWfBlock + (p % 32) * 4 + jm % 4;
            if (p / 32 == item) bits |= kFaceLocal;
        } else {
            const int32_t z = g.g_zone[ids.x - g.nint];
            bits |= ((uint32_t)g.z_dyn[z] & 255u) << 8 | ((uint32_t)g.z_therm[z] & 255u) << 16;
        }
        if (lowmask && ((lowmask[c] >> slot2) & 1u)) bits |= kFaceLow;
        ids.w = (int)bits;
        const double V = g.V[c];
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
            ns[k] = (R)fr.n[k];
            ns2[k] = (R)fr2.n[k];
            og[k] = rec == 1 || !side ? fr.o0[k] : fr.o1[k];
        }
        ns[DIM] = (R)fr.S;
        ns2[DIM] = (R)fr2.S;
        if (grad == 1 && EXACT) {
            const R gp = (R)(fr.S / V);
            og[DIM] = side ? gp : -gp;
            og[DIM + 1] = (R)g.beta[ent >> 1];
        } else if (grad == 1) {  // the values of the gradient pass's table (build_gradient_coefficients)
            const double sv = (side ? 1.0 : -1.0) * (fr.S / V), beta = g.beta[ent >> 1];
            og[DIM] = (R)(side ? beta : 1.0 - beta);
#pragma unroll
            for (int k = 0; k < DIM; ++k) og[DIM + 1 + k] = (R)(sv * fr.n[k]);
        } else if (grad == 2) {  // as gradient_cell forms them (psstGradCalculation.cpp:268-368)
            R lr[7], diff[DIM], w = (R)0;
#pragma unroll
            for (int i = 0; i < (DIM == 2 ? 3 : 7); ++i) lr[i] = (R)g.lsq_r[(int64_t)i * g.nint + c];
#pragma unroll
            for (int k = 0; k < DIM; ++k) {
                diff[k] = (R)g.xc[(int64_t)k * g.nall + ids.y] - (R)g.xc[(int64_t)k * g.nall + c];
                w += diff[k] * diff[k];
            }
            const R ws = (R)1 / w;
            const R al0 = diff[0] / (lr[0] * lr[0]);
            const R al1 = (diff[1] - lr[1] / lr[0] * diff[0]) / (lr[2] * lr[2]);
            R th[DIM];
            th[0] = al0 - lr[1] / lr[0] * al1;
            th[1] = al1;
            if constexpr (DIM == 3) {
                const R al2 = (diff[2] - lr[4] / lr[2] * diff[1] + lr[6] * diff[0]) / (lr[5] * lr[5]);
                th[0] += al2 * lr[6];
                th[1] -= lr[4] / lr[2] * al2;
                th[2] = al2;
            }
#pragma unroll
            for (int k = 0; k < DIM; ++k) og[DIM + k] = ws * th[k];
        }
    }
    uint4 *o = faces + (size_t)blockIdx.x * FD::PIECES * kWfBlock;
    o[t] = make_uint4((uint32_t)ids.x, (uint32_t)ids.y, (uint32_t)ids.z, (uint32_t)ids.w);
#pragma unroll
    for (int i = 0; i < FD::PIECES - 1; ++i) {
        uint4 w;
        memcpy(&w, f + i * FD::PER, 16);
        o[(1 + i) * kWfBlock + t] = w;
    }
    if (round == 0 && q == 0) {
        const double V = c >= 0 ? g.V[c] : 1.0;
        cells[(size_t)item * 32 + slot] = make_double2(V, 1.0 / V);
    }
}

// What a CTA keeps of one of its items between operations: the cells' states by
// stage parity (read by the item's other cells as well, after the CTA barrier
// that begins every operation), their FP64 conservative states at the start of
// the iteration, and per lane and round of four faces the two cells' gradient
// projections. In shared memory for the CTA's first items, in global memory for
// the rest.
template <typename R, int DIM>
struct ItemStore {
    double *w;  // [DIM + 2][32]
    R *own;     // [2][DIM + 3][32]: u.., p, T, rho
    R *proj;    // [rounds][2][DIM + 2][128]: this cell's, the other's
    static __host__ __device__ size_t bytes(int rounds, bool second) {
        return 32 * (DIM + 2) * sizeof(double) + 2 * 32 * (DIM + 3) * sizeof(R) +
               (second ? (size_t)rounds * 2 * (DIM + 2) * kWfBlock * sizeof(R) : 0);
    }
    __device__ __forceinline__ ItemStore(char *p) {
        w = reinterpret_cast<double *>(p);
        own = reinterpret_cast<R *>(w + 32 * (DIM + 2));
        proj = own + 2 * 32 * (DIM + 3);
    }
    __device__ __forceinline__ Prim<R, DIM> state(int s, int slot) const {
        const R *o = own + (s & 1) * 32 * (DIM + 3) + slot;
        Prim<R, DIM> x;
#pragma unroll
        for (int k = 0; k < DIM; ++k) x.u[k] = o[k * 32];
        x.p = o[DIM * 32];
        x.T = o[(DIM + 1) * 32];
        x.rho = o[(DIM + 2) * 32];
        return x;
    }
};

// Norm rows of the CTA's stage operations: every lane puts its component's res^2
// and |res| of its cell here, by operation parity, and during the next operation
// one warp (they take turns) adds them up in a fixed order and writes the row.
template <int NV>
struct NormRows {
    double val[2][2 * NV][33];  // [component][quad of the CTA]
};

// This lane's part of stage operation n's row (NaN contributes nothing to the
// maximum, as in `if (res < |r|)`, psstFiniteVolumeGrid.cpp:331).
template <int NV>
__device__ __forceinline__ void norm_put(NormRows<NV> &rows, unsigned n, double r0, double r1) {
    const int q = threadIdx.x & 3, at = threadIdx.x >> 2;
    double(*v)[33] = rows.val[n & 1u];
    v[q][at] = r0 * r0;
    v[NV + q][at] = fabs(r0) > 0.0 ? fabs(r0) : 0.0;
    if (NV == 5 && q == 0) {
        v[4][at] = r1 * r1;
        v[NV + 4][at] = fabs(r1) > 0.0 ? fabs(r1) : 0.0;
    }
}

// Adds up operation n's row (one warp, after a CTA barrier that followed it).
template <int NV>
__device__ __forceinline__ void norm_write(const NormRows<NV> &rows, unsigned n, double *out) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int c0 = 0; c0 < 2 * NV; c0 += 8) {
        const int c = c0 + (lane >> 2);
        double s = 0.0;
        if (c < 2 * NV) {
            const double *v = rows.val[n & 1u][c] + 8 * (lane & 3);
#pragma unroll
            for (int i = 0; i < 8; ++i) s = c < NV ? s + v[i] : fmax(s, v[i]);
        }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            const double x = __shfl_xor_sync(FULL, s, o);
            s = c < NV ? s + x : fmax(s, x);
        }
        if (c < 2 * NV && (lane & 3) == 0) out[c] = s;
    }
}

// One (item, operation) pair as a lane sees it, and the static data of the lane's
// face in the item's first round: a CTA with one item loads them once (loading
// them every operation took 1640 of 8500 cycles).
template <typename R, int DIM>
struct Lane {
    int32_t c;        // the quad's cell, -1: none
    int item;
    int q, qb, slot;  // lane in the quad, the quad's first lane, the quad's place in the item
    uint4 ids;
    R ns[FaceData<R, DIM>::NS * FaceData<R, DIM>::PER];  // n, S
    double2 vol;
    __device__ __forceinline__ const uint4 *block(const ResSched &w, int r) const {
        return w.faces + ((size_t)item * w.rounds + r) * FaceData<R, DIM>::PIECES * kWfBlock;
    }
    __device__ __forceinline__ void load(const ResSched &w, int it) {
        item = it;
        c = w.cells32[(size_t)it * 32 + slot];
        vol = __ldg(w.cells + (size_t)it * 32 + slot);
        const uint4 *b = block(w, 0);
        ids = __ldg(b + threadIdx.x);
        FaceData<R, DIM>::template fields<0, FaceData<R, DIM>::NS>(b, threadIdx.x, ns);
    }
    // the face of round r: neighbours and flags, n and S
    __device__ __forceinline__ void face(const ResSched &w, int r, uint4 &i, R *f) const {
        constexpr int N = FaceData<R, DIM>::NS;
        if (r == 0) {
            i = ids;
#pragma unroll
            for (int k = 0; k < N * FaceData<R, DIM>::PER; ++k) f[k] = ns[k];
        } else {
            const uint4 *b = block(w, r);
            i = __ldg(b + threadIdx.x);
            FaceData<R, DIM>::template fields<0, N>(b, threadIdx.x, f);
        }
    }
};

// One more attempt of a warp's wait (every lane takes part): whether any lane
// still misses something, after which the caller loads again; `ok` is cleared
// when the wait is given up. The loops around it are the warp's, not the
// lane's: lanes that left a loop of their own one by one would stay apart, and
// every later shuffle would cost 230 cycles more.
__device__ __forceinline__ bool still_waiting(bool miss, bool &ok, Waiter &wt, int where) {
    if (!__any_sync(FULL, miss)) return false;
    const bool more = !__any_sync(FULL, !wt.again(where));
    ok = ok && more;
    return more;
}

// Gradient of the quad's cell. Lane j forms the products of the face at its
// position -- Green-Gauss in the face-loop order (psstGradCalculation.cpp:
// 80-177), least squares in the cell's own order (:268-368; 3D as the corrected
// restatement of gradient_cell) -- and after a transpose lane v adds variable v
// (u.., p, T) over the faces in the reference's order (the fifth variable of 3D
// in every lane), applies the cell limiter and publishes its projection on
// every face's offset.
template <typename R, int DIM, int REC>
__device__ __forceinline__ bool res_gradient(const ResArgs<R> &a, const Lane<R, DIM> &L, const ItemStore<R, DIM> &st, int s,
                                             int k, int where) {
    using FD = FaceData<R, DIM>;
    constexpr int NV = DIM + 2, NP = NV == 5 ? 2 : 1, NS = record_words<R>(DIM + 3), NPS = record_words<R>(NV);
    const DevGrid &g = a.g;
    const int32_t c = L.c;
    const int q = L.q, qb = L.qb, rounds = a.sc.rounds;
    const uint64_t *in = a.state[s & 1];
    uint64_t *proj = a.proj;
    const uint32_t tag = a.tag0 + (uint32_t)s, ptag = a.ptag0 + (uint32_t)k + 1u;
    const bool gg = a.grad == 1;
    bool ok = true;
    Prim<R, DIM> own{};
    own.T = own.p = own.rho = (R)1;  // lanes without a cell: ordinary operands
    R eps2 = (R)0;
    if (c >= 0) {
        own = s == 0 ? unpack<R, DIM>(ldg(a.in + c)) : st.state(s, L.slot);
        if (REC == 2 && a.celllim == 5) eps2 = (R)g.vk_eps2[c];
    }
    R gr[NP][DIM], phi[NP], mx[NP], mn[NP];
    {
        R v[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) v[i] = pvar<R, DIM>(own, i);
        phi[0] = pick<R, 4>(v, q);
        phi[NP - 1] = NP == 2 ? v[NV - 1] : phi[0];
    }
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        mx[i] = mn[i] = phi[i];
#pragma unroll
        for (int t = 0; t < DIM; ++t) gr[i][t] = (R)0;
    }
    for (int r = 0; r < rounds; ++r) {
        uint4 ids;
        R f1[FD::NS * FD::PER], f2[FD::OG * FD::PER];  // n, S; off, g
        L.face(a.sc, r, ids, f1);
        FD::template fields<FD::NS, FD::OG>(L.block(a.sc, r), threadIdx.x, f2);
        const uint32_t bits = ids.w;
        const unsigned valid = __ballot_sync(FULL, (bits & kFaceValid) != 0u);
        if (valid == 0u) break;
        const unsigned vq = valid >> qb;
        const int32_t nb = (int32_t)(gg ? ids.x : ids.y);
        const bool need = (bits & kFaceValid) && s > 0 && nb < g.nint &&
                          !((bits & kFaceLocal) && (gg || (bits & kFaceSame)));
        Record<R, DIM + 3> w;
        Waiter wt{a.sc.sync, a.wk.err, a.wait_ns, 0, 0u};
        const uint64_t *p = in + (size_t)(need ? nb : 0) * NS;
        do {
            if (need) w.fetch(p);
        } while (still_waiting(need && (!w.holds(tag) || a.wait_ns == 0), ok, wt, where));
        if (!ok) return false;
        R oth[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) oth[i] = (R)0;
        if (bits & kFaceValid) {
            if (s == 0 || nb >= g.nint) {
                const Prim<R, DIM> o = unpack<R, DIM>(ld16((s == 0 ? a.in : a.out) + nb));
#pragma unroll
                for (int i = 0; i < NV; ++i) oth[i] = pvar<R, DIM>(o, i);
            } else {
                Prim<R, DIM> x;
                if (need)
                    x = from_record<R, DIM>(w);
                else
                    x = st.state(s, (int)(ids.z % kWfBlock) >> 2);
#pragma unroll
                for (int i = 0; i < NV; ++i) oth[i] = pvar<R, DIM>(x, i);
            }
        }
        if constexpr (sizeof(R) == 4) {
            // as gradient_cell_table: face values in one rounding, summed by fused products
            // with the table's coefficients (products rounded here and then added: errors
            // of u 6% larger after 30 iterations of 3000 tets)
            R tv[NV], d[DIM];
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const R av = pvar<R, DIM>(own, i);
                tv[i] = gg ? fmaf(f2[DIM], oth[i] - av, av) : oth[i] - av;
            }
#pragma unroll
            for (int t = 0; t < DIM; ++t) d[t] = gg ? f2[DIM + 1 + t] : f2[DIM + t];
            const R tv4 = tv[NV - 1];
            quad_transpose(tv, q);
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
                const R y4 = NP == 2 ? __shfl_sync(FULL, tv4, qb + jj) : (R)0;
#pragma unroll
                for (int t = 0; t < DIM; ++t) {
                    const R dj = __shfl_sync(FULL, d[t], qb + jj);
                    if ((vq >> jj) & 1u) {
                        gr[0][t] = fmaf(tv[jj], dj, gr[0][t]);
                        if (NP == 2) gr[NP - 1][t] = fmaf(y4, dj, gr[NP - 1][t]);
                    }
                }
            }
        } else {
            const bool side = bits & kFaceSide;
            const R coef = f2[DIM], beta = f2[DIM + 1];
            R tv[NV];
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const R av = pvar<R, DIM>(own, i);
                if (gg) {
                    const R phi0 = side ? oth[i] : av, phi1 = side ? av : oth[i];
                    tv[i] = (beta * phi0 + ((R)1 - beta) * phi1) * coef;
                } else {
                    tv[i] = oth[i] - av;
                }
            }
#pragma unroll
            for (int t = 0; t < DIM; ++t) {
                const R d = gg ? f1[t] : f2[DIM + t];
                R x[4], x4 = (R)0;
#pragma unroll
                for (int i = 0; i < 4; ++i) x[i] = tv[i] * d;
                if (NP == 2) x4 = tv[NV - 1] * d;
                quad_transpose(x, q);
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    const R y4 = NP == 2 ? __shfl_sync(FULL, x4, qb + jj) : (R)0;
                    if ((vq >> jj) & 1u) {
                        gr[0][t] += x[jj];
                        if (NP == 2) gr[NP - 1][t] += y4;
                    }
                }
            }
        }
        if (REC == 2) {
            R x[4] = {oth[0], oth[1], oth[2], oth[3]};
            quad_transpose(x, q);
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
                const R y4 = NP == 2 ? __shfl_sync(FULL, oth[NV - 1], qb + jj) : (R)0;
                if ((vq >> jj) & 1u) {
                    if (x[jj] > mx[0]) mx[0] = x[jj];
                    if (x[jj] < mn[0]) mn[0] = x[jj];
                    if (NP == 2) {
                        if (y4 > mx[NP - 1]) mx[NP - 1] = y4;
                        if (y4 < mn[NP - 1]) mn[NP - 1] = y4;
                    }
                }
            }
        }
    }
    // offsets of the quad's faces: other lanes' static data, read through L1
    if (REC == 2) {
        R lim[NP];
        // with `div` as the division; false where an operand is out of lin_div's range
        auto limit = [&](auto div) {
            bool fine = true;
#pragma unroll
            for (int i = 0; i < NP; ++i) lim[i] = (R)1;
            for (int r = 0; r < rounds; ++r) {
                const uint4 *block = a.sc.faces + ((size_t)L.item * rounds + r) * FD::PIECES * kWfBlock;
                const int t0 = (int)(threadIdx.x & ~3u);
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    const bool valid = __ldg(block + t0 + jj).w & kFaceValid;
                    R off[FD::OFFP * FD::PER];
                    FD::template fields<FD::NS, FD::OFFP>(block, t0 + jj, off);
#pragma unroll
                    for (int i = 0; i < NP; ++i) {
                        R dm = (R)0;
#pragma unroll
                        for (int t = 0; t < DIM; ++t) dm += gr[i][t] * off[t];
                        const R dp = dm > (R)0 ? mx[i] - phi[i] : mn[i] - phi[i];
                        const bool use = valid && dm != (R)0;
                        const R num = a.celllim == 4 ? dp : (dp * dp + eps2) + (R)2 * dm * dp;
                        const R den = a.celllim == 4 ? dm : dp * dp + (R)2 * dm * dm + dm * dp + eps2;
                        const R d = use ? den : (R)1;
                        fine = fine && den_ok(d) && zero_or_in_range(num);
                        R pf = div(num, d);
                        if (a.celllim == 4) pf = pf < (R)1 ? pf : (R)1;
                        if (use && pf < lim[i]) lim[i] = pf;
                    }
                }
            }
            return fine;
        };
        if (!limit([](R x, R y) { return lin_div(x, y); }) && c >= 0) limit([](R x, R y) { return x / y; });
#pragma unroll
        for (int i = 0; i < NP; ++i)
#pragma unroll
            for (int t = 0; t < DIM; ++t) gr[i][t] = gr[i][t] * lim[i];
    }
    for (int r = 0; r < rounds; ++r) {
        const size_t lb = (size_t)L.item * rounds + r;
        const uint4 *block = a.sc.faces + lb * FD::PIECES * kWfBlock;
        const int t0 = (int)(threadIdx.x & ~3u);
        R *pj = st.proj + (size_t)r * 2 * NV * kWfBlock;
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
            const uint32_t bits = __ldg(block + t0 + jj).w;
            if (!(bits & kFaceInner)) continue;  // boundary faces take the ghost's physical flux
            R off[FD::OFFP * FD::PER];
            FD::template fields<FD::NS, FD::OFFP>(block, t0 + jj, off);
#pragma unroll
            for (int i = 0; i < NP; ++i) {
                R d = (R)0;
#pragma unroll
                for (int t = 0; t < DIM; ++t) d += gr[i][t] * off[t];
                if (i == 1 && q != 0) continue;
                pj[(i == 0 ? q : NV - 1) * kWfBlock + t0 + jj] = d;
            }
        }
        // each lane publishes its own face's projections to another item's cell
        __syncwarp();
        const uint32_t mine = __ldg(block + threadIdx.x).w;
        if ((mine & (kFaceInner | kFaceLocal)) == kFaceInner) {
            R v[NV];
#pragma unroll
            for (int i = 0; i < NV; ++i) v[i] = pj[i * kWfBlock + threadIdx.x];
#pragma unroll
            for (int h = 0; h < NPS / 4; ++h) publish_sector<R, NV>(proj + (lb * kWfBlock + threadIdx.x) * NPS, h, v, ptag);
        }
    }
    if (c >= 0 && k == a.n_iter - 1) {  // the gradients that psst_solver_get_array reads
        GradRec<R, DIM> *o = reinterpret_cast<GradRec<R, DIM> *>(a.wk.grec) + c;
#pragma unroll
        for (int t = 0; t < DIM; ++t) {
            o->g[q * DIM + t] = gr[0][t];
            if (NP == 2 && q == 0) o->g[(NV - 1) * DIM + t] = gr[NP - 1][t];
        }
    }
    return true;
}

// RK stage `stage` of iteration k (stage s of the call) of the quad's cell.
// Lane q takes the faces q, q + 4, .. in the face-loop order for the fluxes
// (psstConvectiveFlow.cpp:289-299 as a per-cell sum) and those of the cell's own
// order for the local time step (psstLocalTimeCalculation.cpp:90-131, 175-213;
// in the sequential mode neighbours updated earlier in the reference's order
// are read from this stage's results); RK update and primitives
// (psstFiniteVolumeGrid.cpp:324-346) one component per lane, ghosts (:351-366)
// by the lane of their face.
template <typename R, int DIM, int REC, int LIM>
__device__ __forceinline__ bool res_stage(const ResArgs<R> &a, const Lane<R, DIM> &L, const ItemStore<R, DIM> &st, int s, int k,
                                          int stage, int where, NormRows<DIM + 2> &rows, unsigned nrow) {
    using FD = FaceData<R, DIM>;
    constexpr int NV = DIM + 2, NW = DIM + 3, NS = record_words<R>(NW), NPS = record_words<R>(NV);
    constexpr bool EXACT = sizeof(R) == 8;
    const DevGrid &g = a.g;
    const int32_t c = L.c;
    const int q = L.q, qb = L.qb, rounds = a.sc.rounds;
    const uint64_t *in = a.state[s & 1];
    uint64_t *next = a.state[(s + 1) & 1];
    const uint64_t *proj = a.proj;
    const CellRec<R> *ghost = s == 0 ? a.in : a.out;
    const uint32_t tag = a.tag0 + (uint32_t)s, ptag = a.ptag0 + (uint32_t)k + 1u;
    const bool first = stage == 0, last = stage == a.nst - 1, end = s == a.nops_stage - 1;
    const R grm = (R)a.gas.gamma * (R)a.gas.rm;
    bool ok = true;
    Prim<R, DIM> own{};
    own.T = own.p = own.rho = (R)1;  // lanes without a cell: ordinary operands
    double pw = 1.0, pw4 = 1.0;
    const double2 vol = L.vol;
    if (c >= 0) {
        if (s == 0) {
            own = unpack<R, DIM>(ldg(a.in + c));
            pw = a.wk.w[(int64_t)q * g.nint + c];
            st.w[q * 32 + L.slot] = pw;
            if (NV == 5) {
                pw4 = a.wk.w[(int64_t)4 * g.nint + c];
                if (q == 0) st.w[4 * 32 + L.slot] = pw4;
            }
        } else {
            own = st.state(s, L.slot);
            pw = st.w[q * 32 + L.slot];
            if (NV == 5) pw4 = st.w[4 * 32 + L.slot];
        }
    }
    R cc = lin_sqrt(grm * own.T);
    if (!positive_in_range<100, 100>(grm * own.T)) cc = sqrt(grm * own.T);
    // whether a cell of another item reads this one (out of the face-loop order,
    // cells of the same item read the published states as well)
    bool outside = a.sc.seq || !a.sc.same_order;
    R res = (R)0, res4 = (R)0, den = (R)0, nnb = (R)0, area[DIM];
#pragma unroll
    for (int t = 0; t < DIM; ++t) area[t] = (R)0;
    for (int r = 0; r < rounds; ++r) {
        uint4 ids;
        R f[FD::NS * FD::PER], f2[FD::NS * FD::PER];  // n, S of the face; of the own-order face
        L.face(a.sc, r, ids, f);
        if (a.sc.same_order) {
#pragma unroll
            for (int i = 0; i <= DIM; ++i) f2[i] = f[i];
        } else {
            FD::template fields<FD::NS + FD::OG, FD::NS>(L.block(a.sc, r), threadIdx.x, f2);
        }
        const uint32_t bits = ids.w;
        const unsigned valid = __ballot_sync(FULL, (bits & kFaceValid) != 0u);
        if (valid == 0u) break;
        const unsigned vq = valid >> qb;
        const bool side = bits & kFaceSide, inner = bits & kFaceInner;
        const int32_t nb = (int32_t)ids.x, nb2 = (int32_t)ids.y;
        R *pj = st.proj + (size_t)r * 2 * NV * kWfBlock + threadIdx.x;
        const bool local = bits & kFaceLocal;
        const unsigned far = __ballot_sync(FULL, inner && !local);  // every lane takes part, whatever `outside` is
        outside = outside || (far >> qb & 15u) != 0u;
        Record<R, NV> rp;
        Record<R, NW> w1, w2;
        // what this lane has to wait for: a cell across in another item, its
        // projections (once an iteration), and for the time step the own-order
        // neighbour where it is another one or has to be of this stage already
        const bool low = a.lc == 1 && (bits & kFaceLow);
        const bool apart = a.lc == 1 && (bits & kFaceValid) && !(bits & kFaceSame) && !low;
        const bool need1 = inner && !local && s > 0, needp = REC != 0 && inner && !local && first;
        const bool need2 = low || (apart && s > 0 && nb2 < g.nint);
        const uint32_t tag2 = low ? tag + 1u : tag;
        const uint64_t *p1 = in + (size_t)nb * NS, *pp = proj + (size_t)ids.z * NPS;
        const uint64_t *p2 = (low ? next : in) + (size_t)nb2 * NS;
        Waiter wt{a.sc.sync, a.wk.err, a.wait_ns, 0, 0u};
        bool miss1 = need1, missp = needp, miss2 = need2;
        do {
            if (miss1) w1.fetch(p1);
            if (missp) rp.fetch(pp);
            if (miss2) w2.fetch(p2);
            if (a.wait_ns != 0) {
                miss1 = miss1 && !w1.holds(tag);
                missp = missp && !rp.holds(ptag);
                miss2 = miss2 && !w2.holds(tag2);
            }
        } while (still_waiting(miss1 || missp || miss2, ok, wt, where));
        if (!ok) return false;
        if (REC != 0 && inner && first) {
            const int lane = (int)(ids.z % kWfBlock);
            const R *there = st.proj + (size_t)((int)(ids.z / kWfBlock) % rounds) * 2 * NV * kWfBlock + lane;
#pragma unroll
            for (int v = 0; v < NV; ++v) pj[(NV + v) * kWfBlock] = local ? there[v * kWfBlock] : rp.value(v);
        }
        Prim<R, DIM> oth = own, on;
        if (need1)
            oth = from_record<R, DIM>(w1);
        else if (local && s > 0)
            oth = st.state(s, (int)(ids.z % kWfBlock) >> 2);
        else if (bits & kFaceValid)
            oth = unpack<R, DIM>(ld16(ghost + nb));
        on = oth;
        if (need2)
            on = from_record<R, DIM>(w2);
        else if (apart)
            on = unpack<R, DIM>(ld16(ghost + nb2));
        // the face's flux (times area, signed for this cell); a boundary face has
        // the ghost on its side `edge`
        R o[NV], pu[DIM];
        {
            const int edge = inner ? -1 : side ? 0 : 1;
            Prim<R, DIM> rr[2];
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const R ov = pvar<R, DIM>(oth, i), wv = pvar<R, DIM>(own, i);
                pvar<R, DIM>(rr[0], i) = side ? ov : wv;
                pvar<R, DIM>(rr[1], i) = side ? wv : ov;
            }
            rr[0].rho = side ? oth.rho : own.rho;
            rr[1].rho = side ? own.rho : oth.rho;
            bool exact = true;
            R e0[NV], e1[NV];
            if (REC) {
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    const R d0 = inner ? pj[v * kWfBlock] : (R)0, dd = inner ? pj[(NV + v) * kWfBlock] : (R)0;
                    e0[v] = side ? dd : d0;
                    e1[v] = side ? d0 : dd;
                }
                Prim<R, DIM> x[2] = {rr[0], rr[1]};
                lin_reconstruct<R, DIM, REC, LIM>(x, e0, e1, (R)a.gas.rm, exact);
                // boundary faces keep the cells' own values (zero projections, own density)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const R rho = rr[h].rho;
                    rr[h] = x[h];
                    rr[h].rho = inner ? x[h].rho : rho;
                }
            }
            R flow[NV];
            if (a.flux == 1)
                lin_flux<R, DIM, 1>(rr, f, a.gas, edge, flow, exact);
            else if (a.flux == 2)
                lin_flux<R, DIM, 2>(rr, f, a.gas, edge, flow, exact);
            else
                lin_flux<R, DIM, 3>(rr, f, a.gas, edge, flow, exact);
            if (!exact && (bits & kFaceValid)) {
                PlainFace<R, DIM, REC, LIM> pf;
                pf.r[0] = side ? oth : own;
                pf.r[1] = side ? own : oth;
                pf.flux = a.flux;
                pf.edge = edge;
                if (REC)
#pragma unroll
                    for (int v = 0; v < NV; ++v) {
                        pf.d0[v] = e0[v];
                        pf.d1[v] = e1[v];
                    }
#pragma unroll
                for (int t = 0; t < DIM; ++t) pf.n[t] = f[t];
                const bool ordered = PlainFace<R, DIM, REC, LIM>::run(&pf, &a.gas);
                if (!ordered) flag_error(a.wk.err, a.flux == 2 ? ERR_HLL : ERR_HLLC, c);
#pragma unroll
                for (int v = 0; v < NV; ++v) flow[v] = ordered ? pf.flow[v] : (R)0;
            }
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const R x = flow[v] * f[DIM];
                o[v] = side ? x : -x;
            }
        }
        // the time step's terms of this face: products in the reference's
        // expressions, the running sums below
        const R sj = f2[DIM];
        R nv = (R)0, cn = (R)0;
        if (a.lc == 1) {
            R cs = lin_sqrt(grm * on.T);
            if (!positive_in_range<100, 100>(grm * on.T)) cs = sqrt(grm * on.T);
            cn = (cs + cc) * (R)0.5;
        }
#pragma unroll
        for (int t = 0; t < DIM; ++t) {
            nv += own.u[t] * f2[t];
            pu[t] = a.lc == 2 ? sj * fabs(f2[t]) : on.u[t] * f2[t];
        }
        // in the reference's order over the round's faces: lane v the residual's
        // component v (the fifth: every lane) ...
        const R o4 = NV == 5 ? o[NV - 1] : (R)0;
        quad_transpose(o, q);
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
            const R x4 = NV == 5 ? __shfl_sync(FULL, o4, qb + jj) : (R)0;
            if ((vq >> jj) & 1u) {
                res += o[jj];
                if (NV == 5) res4 += x4;
            }
        }
        // ... and the time step, each lane its own face's term of the chain
        if (a.lc == 1) {
            R mine = (R)0;
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
                R t = nnb;
#pragma unroll
                for (int d = 0; d < DIM; ++d) t += pu[d];
                t = (t + nv) * (R)0.5;
                if (jj == q) mine = t;
                t = __shfl_sync(FULL, t, qb + jj);
                if ((vq >> jj) & 1u) nnb = t;
            }
            const R term = (fabs(mine) + cn) * sj;
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
                const R x = __shfl_sync(FULL, term, qb + jj);
                if ((vq >> jj) & 1u) den += x;
            }
        } else if (a.lc == 2) {
#pragma unroll
            for (int jj = 0; jj < 4; ++jj)
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    const R x = __shfl_sync(FULL, pu[d], qb + jj);
                    if ((vq >> jj) & 1u) area[d] += x;
                }
        }
    }
    if (a.lc == 2) {
#pragma unroll
        for (int d = 0; d < DIM; ++d) den += (fabs(own.u[d]) + cc) * area[d] * (R)0.5;
    }
    // time step, RK update and primitives: lane v component v (3D: every lane the
    // energy as well), with `quot(x, d, 1 / d)` as the division
    const double alpha = a.alpha[stage];
    const R num = (R)a.cfl * (R)vol.x;
    double dt, w, w4, rho, u[DIM], T;
    auto update = [&](auto plain) {
        constexpr bool P = decltype(plain)::value;
        auto over = [](double x, double d, double y) { return P ? x / d : lin_quot(x, d, y); };
        dt = a.dt_uniform;
        if (a.lc != 0) dt = (double)(P ? num / den : lin_div(num, den));
        const double x = dt * alpha * (double)res, x4 = dt * alpha * (double)res4;
        if (EXACT) {
            w = pw - over(x, vol.x, vol.y);
            w4 = NV == 5 ? pw4 - over(x4, vol.x, vol.y) : 0.0;
        } else {
            const double step = over(dt * alpha, vol.x, vol.y);
            w = pw - step * (double)res;
            w4 = NV == 5 ? pw4 - step * (double)res4 : 0.0;
        }
        rho = __shfl_sync(FULL, w, qb + DIM);
        const double y = P ? 1.0 / rho : lin_recip(rho);
        const double quot = EXACT ? over(w, rho, y) : w * y;
        double vs = 0.0;
#pragma unroll
        for (int t = 0; t < DIM; ++t) {
            u[t] = __shfl_sync(FULL, quot, qb + t);
            vs += u[t] * u[t];
        }
        const double e = NV == 5 ? (EXACT ? over(w4, rho, y) : w4 * y) : __shfl_sync(FULL, quot, qb + 3);
        const double z = e - (vs * 0.5);
        T = EXACT ? over(z, a.gas.cv, a.rcv) : z * a.rcv;
        return den_ok(vol.x) && den_ok(rho) && den_ok(a.gas.cv) && zero_or_in_range(x) && zero_or_in_range(x4) &&
               zero_or_in_range(w) && zero_or_in_range(w4) && zero_or_in_range(z) &&
               (a.lc == 0 || (den_ok(den) && zero_or_in_range(num)));
    };
    if (!__all_sync(FULL, update(std::false_type()) || c < 0)) update(std::true_type());
    const double p = rho * a.gas.rm * T;
    Prim<R, DIM> nw;
    nw.p = (R)p;
    nw.T = (R)T;
    nw.rho = (R)rho;
#pragma unroll
    for (int t = 0; t < DIM; ++t) nw.u[t] = (R)u[t];
    if (c >= 0) {
        R v[NW];
#pragma unroll
        for (int i = 0; i < NV; ++i) v[i] = pvar<R, DIM>(nw, i);
        v[NV] = nw.rho;
        // the last stage as well: later neighbours of the sequential order read it
        if (outside && q < NS / 4) publish_sector<R, NW>(next + (size_t)c * NS, q, v, tag + 1u);
        R *o = st.own + ((s + 1) & 1) * 32 * NW + L.slot;
        o[q * 32] = pick<R, 4>(v, q);
        if (q < NW - 4) o[(4 + q) * 32] = q == 0 ? v[4] : v[NW - 1];
        if (last) {
            st.w[q * 32 + L.slot] = w;
            if (NV == 5 && q == 0) st.w[4 * 32 + L.slot] = w4;
        }
        // ghosts of this lane's boundary faces
        for (int r = 0; r < rounds; ++r) {
            uint4 ids;
            R n[FD::NS * FD::PER];
            L.face(a.sc, r, ids, n);
            if ((ids.w & (kFaceValid | kFaceInner)) != kFaceValid) continue;
            st16(a.out + (int32_t)ids.x,
                 ghost_from<R, DIM>(ld16(ghost + (int32_t)ids.x), nw, (int)(ids.w >> 8 & 255u),
                                    (int)(ids.w >> 16 & 255u), n, a.gas));
        }
        const double rv = (double)res, rv4 = (double)res4;
        if (!(rv - rv == 0.0) || (NV == 5 && !(rv4 - rv4 == 0.0))) flag_error(a.wk.err, ERR_NONFINITE_RES, c);
        if (q == 0 && !(rho > 0.0 && T > 0.0)) flag_error(a.wk.err, ERR_BAD_STATE, c);
        if (end) {
            a.wk.w[(int64_t)q * g.nint + c] = w;
            if (NV == 5 && q == 0) a.wk.w[(int64_t)4 * g.nint + c] = w4;
            if (q == 0) {
                a.wk.dt[c] = dt;
                st16(a.out + c, pack<R, DIM>(nw.p, nw.T, nw.rho, nw.u));
            }
        }
    }
    norm_put<NV>(rows, nrow, c >= 0 ? (double)res : 0.0, c >= 0 ? (double)res4 : 0.0);
    return true;
}

// Residual columns of the iterations it = block, block + grid, ..: per stage the
// RMS over the cells and the max |res|, then the max over stages (the reference's
// column, psstFiniteVolumeGrid.cpp:331-332; the RMS column is this project's).
// Rows are added in a fixed order.
template <int NV, typename R>
__device__ __forceinline__ void res_columns(const ResArgs<R> &a) {
    constexpr int W = 2 * NV, G = kWfBlock / W;
    __shared__ double red[G * W];
    const int t = threadIdx.x, comp = t % W, grp = t / W;
    for (int64_t it = blockIdx.x; it < a.n_iter; it += gridDim.x) {
        double col = 0.0;
        for (int stage = 0; stage < a.nst; ++stage) {
            const double *p = a.sc.rows + ((it * a.nst + stage) * a.sc.nitems) * W;
            double v = 0.0;
            if (t < G * W)
                for (int i = grp; i < a.sc.nitems; i += G) {
                    const double x = ldcg(p + (size_t)i * W + comp);
                    v = comp < NV ? v + x : fmax(v, x);
                }
            if (t < G * W) red[t] = v;
            __syncthreads();
            if (t < W) {
                double x = 0.0;
                for (int i = 0; i < G; ++i) x = comp < NV ? x + red[i * W + t] : fmax(x, red[i * W + t]);
                if (t < NV) x = sqrt(x / (double)(a.g.nint > 0 ? a.g.nint : 1));
                col = fmax(col, x);
            }
            __syncthreads();
        }
        if (t < NV) a.wk.l2[it * NV + t] = col;
        else if (t < W) a.wk.linf[it * NV + t - NV] = col;
    }
}

// Two builds of the kernel: few CTAs an SM with the registers the code wants, and
// one more an SM with some spilled, for meshes that need that many CTAs to have
// one item each (a second item doubles an operation).
template <typename R, int DIM, bool MORE>
constexpr int res_min_blocks() {
    return sizeof(R) == 4 ? (MORE ? 5 : 4) : DIM == 2 && MORE ? 3 : 2;
}

template <typename R, int DIM, int REC, int LIM, bool MORE>
__global__ void __launch_bounds__(kWfBlock, res_min_blocks<R, DIM, MORE>()) k_resident(const __grid_constant__ ResArgs<R> a) {
    constexpr int NV = DIM + 2;
    extern __shared__ __align__(16) char res_smem[];
    __shared__ NormRows<NV> rows;
    const ResSched &w = a.sc;
    const int o0 = w.own_ptr[blockIdx.x], o1 = w.own_ptr[blockIdx.x + 1];
    const size_t ibytes = ItemStore<R, DIM>::bytes(w.rounds, REC != 0);
    Lane<R, DIM> L;
    L.item = -1;
    L.q = (int)threadIdx.x % kWfLanes;
    L.slot = (int)threadIdx.x / kWfLanes;
    L.qb = ((int)threadIdx.x & 31) & ~(kWfLanes - 1);
    const int gofs = a.nopi - a.nst;
    const int2 it0 = w.own[o0];
    unsigned nrow = 0u;
    double *row = nullptr;  // where the last stage operation's row goes
    // ok: this warp's waits so far; go: every warp's, as of the last CTA barrier.
    // A warp that gave up still meets the others at their next barrier, and all
    // of them leave there (the CTA's barriers stay in step).
    bool ok = true, go = true;
    const int turns = a.nops + w.max_turn;
    for (int mb = 0; go && mb < turns; ++mb)
        for (int x = o0; go && x < o1; ++x) {
            const int2 it = x == o0 ? it0 : w.own[x];  // item, turn = level / period
            const int m = mb - it.y;
            if (m < 0 || m >= a.nops) continue;
            const int k = m / a.nopi, j = m - k * a.nopi;
            if (L.item != it.x) L.load(w, it.x);
            const int idx = x - o0;
            const ItemStore<R, DIM> st(idx < w.smem_items ? res_smem + idx * ibytes
                                                          : w.store + (size_t)it.x * ibytes);
            go = __syncthreads_and(ok);  // the CTA's previous operation is complete
            if (!go) break;
            if (j < gofs) {
                if constexpr (REC != 0) ok = res_gradient<R, DIM, REC>(a, L, st, k * a.nst, k, m);
            } else {
                const int s = k * a.nst + (j - gofs);
                ok = res_stage<R, DIM, REC, LIM>(a, L, st, s, k, j - gofs, m, rows, nrow);
                if (nrow > 0u && (nrow & 3u) == threadIdx.x >> 5) norm_write<NV>(rows, nrow - 1u, row);
                row = w.rows + ((size_t)s * w.nitems + it.x) * 2 * NV;
                ++nrow;
            }
        }
    if (go) go = __syncthreads_and(ok);
    if (go && nrow > 0u && threadIdx.x < 32) norm_write<NV>(rows, nrow - 1u, row);
    // every CTA done: the columns of this CTA's share of the iterations
    __shared__ int s_go;
    __syncthreads();
    if (threadIdx.x == 0) {
        if (go) {
            __threadfence();
            atomicAdd(&w.sync[0], 1u);
            Waiter wt{w.sync, a.wk.err, a.wait_ns, 0, 0u};
            while (go && (int)(ld_acquire_gpu(&w.sync[0]) - w.arrive_target) < 0) go = wt.again(a.nops);
        }
        s_go = go;
    }
    __syncthreads();
    if (s_go) res_columns<NV, R>(a);
}

template <typename R, int DIM, int REC, int LIM>
cudaError_t res_launch(const ResArgs<R> &a, int nblocks, bool more, size_t smem, cudaStream_t s) {
    void *args[] = {const_cast<ResArgs<R> *>(&a)};
    const void *kern = more ? reinterpret_cast<const void *>(&k_resident<R, DIM, REC, LIM, true>)
                            : reinterpret_cast<const void *>(&k_resident<R, DIM, REC, LIM, false>);
    return cudaLaunchCooperativeKernel(kern, dim3(nblocks), dim3(kWfBlock), args, smem, s);
}

// Most co-resident CTAs with the most items kept in shared memory (at most
// want): keeping the item on chip comes after having another CTA.
template <typename R, int DIM, int REC, int LIM>
int res_max_blocks(int rounds, bool more, int want, int *items, size_t *smem) {
    int dev = 0, nsm = 0, lim = 0;
    auto kern = more ? k_resident<R, DIM, REC, LIM, true> : k_resident<R, DIM, REC, LIM, false>;
    cudaFuncAttributes at{};
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 0;
    if (cudaFuncGetAttributes(&at, kern) != cudaSuccess) return 0;
    lim -= (int)at.sharedSizeBytes;  // the kernel's own limit, the same for every solver
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) != cudaSuccess) return 0;
    const size_t per = ItemStore<R, DIM>::bytes(rounds, REC != 0);
    int best = 0;
    for (int n = 0; n <= want && n * per <= (size_t)lim; ++n) {
        int occ = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kWfBlock, n * per) != cudaSuccess) return 0;
        if (occ < best) break;
        best = occ;
        *items = n;
        *smem = n * per;
    }
    return best * nsm;
}

}  // namespace psst
