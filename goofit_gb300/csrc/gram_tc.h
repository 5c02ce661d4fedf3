// Device code of the normalisation integrals on the 5th-generation tensor cores (tcgen05.mma, kind::tf32), part of
// the source generated for trees with amplitude nodes (mixed engine).
//
// The generated kernel gf_ampng evaluates the amplitudes of the normalisation points and contracts them in the same
// pass: with x_i the 2C real columns of a point (Re X_0, Im X_0, Re X_1, ...: the values, then the derivatives) and
// e its efficiency it sums
//     G_ij = sum_p x_i(p) e(p) x_j(p),   i < 2C, j < 2n (n values),
// from which the host forms I_ab = sum_p X_a conj(X_b) e and the derivative rows H.  It takes the place of the
// reference's one launch per entry (src/PDFs/physics/detail/SpecialResonanceIntegrator.cu:52-121,
// src/PDFs/physics/detail/NormIntegrator.cu:15-68).
//
// Why one pass: the columns never reach HBM.  With 2e6 four-body events and 30 columns they were 480 MB written by one
// kernel (216 us) and read by a second (486 us, bound by the issue of its copy, split and drain, with one CTA of 8
// warps per SM); with 794,107 Dalitz points and 16 columns 92 + 103 us.
//
// One CTA of 128 threads takes 128 points at a time, one per thread.  A thread splits its point's values into TF32
// pairs, x = hi + lo, and stores them K-major (the point index is K) in the 128-byte swizzled layout: the 32 lanes of
// a warp are 32 consecutive points, so each store fills one 128-byte row and no bank twice.  The MMA's 128 rows are
// S = 128 / W slices of W >= 2C real columns, each slice W of the 128 points, and its N = S Wn columns are the slices'
// value columns (Wn: 2n rounded up to 8).  Blocks of D that pair two slices are products of unrelated points and are
// never read.  The value columns of B are rows of A where no efficiency weighs them (Amp4Body): rows are then ordered
// by (group of 8 columns, slice), which makes them A's first N rows, and 64 KB hold a CTA's operands, so that three
// CTAs stay resident.  Weighted (Amp3Body), B = e x has its own 1024 Wn bytes.
//
// Each product takes four MMAs (lo lo + hi lo + lo hi + hi hi).  The tensor core's FP32
// accumulation rounds towards zero, so an accumulator sums one tile's 32 points per slice only: the small terms first,
// then four MMAs of large ones.  That leaves sums of squares 8 to 9e-8 short; without lo lo, which is positive in each of
// them, it was 12 to 13e-8 (8 resonances, 794,107 points, the error of a fit's NLL against 64 bits 4.1e-7 -> 3.1e-7).  The tile's accumulator is added to a compensated FP32 pair per entry, which lives in
// tensor memory beside it (registers would cost the amplitudes their occupancy).  The MMAs of one tile run while the
// threads evaluate the amplitudes of the next, so one operand buffer is enough.
//
// Every wait is bounded: after a wait that runs out the CTA stops issuing work, waits (bounded) for what it issued, frees
// its tensor memory and writes kGramStopped in the place of its partials, and the sums hand it on.  The host may read the
// sums while the launch ends, so the failure has to stand in the words that it waits for: a flag beside them, written by
// another kernel, need not be visible when they are.
#pragma once

#include <cstddef>

namespace gf {

constexpr int kGramThreads = 128;
// the partials of a CTA whose wait ran out, and the sums over them: a signalling NaN, which no arithmetic gives
constexpr unsigned long long kGramStopped = 0x7ff40000dead0002ull;

// real columns per slice for a node of nc complex columns (0: more than 64 real columns, no tensor-core kernel) and
// value columns per slice for n amplitudes
inline int gram_width(int nc) { return 2 * nc <= 32 ? 32 : 2 * nc <= 64 ? 64 : 0; }
inline int gram_values(int n) { return (2 * n + 7) / 8 * 8; }
// tensor-memory columns: the accumulators (one per 32 points of a slice), the pairs; allocated as a power of two
inline int gram_tmem(int w, int wn) {
    const int need = w / 32 * (128 / w) * wn + 2 * wn;
    int c          = 32;
    while(c < need)
        c *= 2;
    return c;
}
// dynamic shared memory: the operands in 1024-byte aligned blocks, and never less than what keeps the CTAs of an SM
// (228 KB) from asking for more than its 512 tensor-memory columns: a CTA that had to wait for them would stay idle
inline size_t gram_smem(int w, int wn, bool weighted) {
    const size_t ops   = 1024 + 2 * (size_t)(w / 32) * 128 * 128 + (weighted ? (size_t)1024 * wn : 0);
    const size_t share = (size_t)228 * 1024 / (512 / gram_tmem(w, wn) + 1) + 1;
    return ops > share ? ops : share;
}

const char *const kGramSource = R"CUDA(
#define GF_GRAM_STOPPED 0x7ff40000dead0002ull /* kGramStopped */
__device__ __forceinline__ unsigned gf_s32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void gf_tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void gf_tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// x rounded to TF32 (11 significant bits, ties away from zero) by integer operations; x - gf_tf32(x) is exact in
// FP32, and the tensor core reads it truncated to TF32
__device__ __forceinline__ float gf_tf32(float x) { return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xFFFFE000u); }
// 8 consecutive FP32 columns of this thread's tensor-memory lane; v holds them once gf_tmem_got has waited and has
// been given v (so that no use of v moves above the wait)
__device__ __forceinline__ void gf_tmem_ld8(unsigned addr, float *v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "r"(addr) : "memory");
}
__device__ __forceinline__ void gf_tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void gf_tmem_got(float *v) {
    asm volatile("" : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7]));
}
__device__ __forceinline__ void gf_tmem_st8(unsigned addr, const float *v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(addr),
                 "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
                 "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
                 "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])) : "memory");
}
__device__ __forceinline__ void gf_tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// One lane of a converged warp.  Issuing a tile's MMAs is on the path of all its threads, which meet before and
// after it; from an elected lane it is shorter than from threadIdx.x == 0 (rebuild of 8 resonances 395 -> 379 us, of the
// four-body model 928 -> 892 us), and each 32-point block of a slice has its own warp issue its 16 MMAs, to its own
// accumulator (four-body, two blocks: 892 -> 835 us).
__device__ __forceinline__ bool gf_elect() {
    unsigned p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
struct GfGramShared {
    unsigned long long mbar, never; /* MMAs of a tile (a commit per block); a barrier that nothing arrives on (test of the failure path) */
    unsigned tmem;
};

// NC complex columns, NA of them values; W, WN, WT as above; COLS tensor-memory columns
template <int W, int WN, bool WT, int NC, int NA, int COLS>
struct GfGram {
    static constexpr int S = 128 / W, N = S * WN, KB = W / 32;
    static constexpr unsigned ABYTES = KB * 16384u, BBYTES = KB * N * 128u, H = KB * N, L = KB * N + WN;
    // instruction descriptor of kind::tf32: D FP32 (bits 4-5), A and B TF32 (bits 7-9, 10-12), both K-major, N >> 3 in
    // bits 17-22, M >> 4 in bits 24-28
    static constexpr unsigned IDESC = (1u << 4) | (2u << 7) | (2u << 10) | ((unsigned)(N >> 3) << 17) | (8u << 24);
    GfGramShared *sh;
    unsigned char *ops;
    unsigned base, store, storeB, tmem;
    unsigned long long limit;
    int stall, last; /* last: the tile whose MMAs were committed last, -1: none */
    // row of A (and lane of D) and column of D of (slice s, column i)
    static __device__ __forceinline__ int rowOf(int s, int i) { return WT ? s * W + i : (i >> 3) * 8 * S + s * 8 + (i & 7); }

    __device__ __forceinline__ GfGram(const GfArgs &a, GfGramShared *shared, unsigned char *dyn) : sh(shared) {
        const int tid = threadIdx.x, s = tid / W, k = tid % W;
        base = (gf_s32(dyn) + 1023u) & ~1023u;
        ops  = dyn + (base - gf_s32(dyn));
        // this thread's point k of slice s: its 32-point block, 16-byte chunk (swizzled by the row's low bits below)
        const unsigned kk = ((unsigned)((k >> 2) & 7) << 4) + (unsigned)(k & 3) * 4u;
        store  = base + (unsigned)(k >> 5) * 16384u + (unsigned)rowOf(s, 0) * 128u + kk;
        storeB = base + 2 * ABYTES + (unsigned)(k >> 5) * (N * 128u) + (unsigned)(s * WN) * 128u + kk;
        limit  = a.gram_ns;
        stall  = a.gram_stall;
        last   = -1;
        for(unsigned i = tid; i < (2 * ABYTES + (WT ? 2 * BBYTES : 0u)) / 16; i += 128) // padding rows stay zero
            reinterpret_cast<uint4 *>(ops)[i] = make_uint4(0u, 0u, 0u, 0u);
        if(tid == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(gf_s32(&sh->mbar)), "r"(KB) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(gf_s32(&sh->never)) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        if(tid < 32) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(gf_s32(&sh->tmem)), "r"(COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
        gf_tc_before();
        __syncthreads();
        gf_tc_after();
        tmem = sh->tmem;
        const float z[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for(int j = 0; j < 2 * WN; j += 8)
            gf_tmem_st8(lane() + H + j, z);
        gf_tmem_wait_st();
    }
    // tensor-memory address of this warp's 32 lanes
    __device__ __forceinline__ unsigned lane() const { return tmem + ((threadIdx.x & 96u) << 16); }
    // waits for the MMAs of tile u; the same answer in all lanes of a warp
    __device__ __forceinline__ bool wait(int u) {
        bool ok = gf_mbar_wait(&sh->mbar, (unsigned)(u & 1), limit);
        if(u == stall)
            ok = ok && gf_mbar_wait(&sh->never, 0u, limit);
        return __all_sync(0xffffffffu, ok);
    }
    // adds the finished tile's accumulators to the pairs
    __device__ __forceinline__ void drain() {
        gf_tc_after();
        const int row = threadIdx.x, s = WT ? row / W : (row >> 3) % S;
#pragma unroll
        for(int j = 0; j < WN; j += 8) {
            // with S slices in a warp (rows of an unweighted node) the lanes keep their own slice's columns; one load
            // at a time (all in flight before one wait took 2 x 48 registers and made the kernel 13% slower)
            constexpr int Q = WT ? 1 : S;
            float h[8], l[8];
            gf_tmem_ld8(lane() + H + j, h);
            gf_tmem_ld8(lane() + L + j, l);
            gf_tmem_wait_ld();
            gf_tmem_got(h);
            gf_tmem_got(l);
#pragma unroll
            for(int b = 0; b < KB; ++b) {
                float v[8];
#pragma unroll
                for(int q = 0; q < Q; ++q) {
                    float w[8];
                    gf_tmem_ld8(lane() + (unsigned)(b * N + (WT ? s * WN + j : j * S + q * 8)), w);
                    gf_tmem_wait_ld();
                    gf_tmem_got(w);
#pragma unroll
                    for(int i = 0; i < 8; ++i)
                        v[i] = q == 0 || q == s ? w[i] : v[i];
                }
#pragma unroll
                for(int i = 0; i < 8; ++i) {
                    const float x = v[i], t = h[i] + x, bp = t - h[i];
                    l[i] += (h[i] - (t - bp)) + (x - bp);
                    h[i] = t;
                }
            }
            gf_tmem_st8(lane() + H + j, h);
            gf_tmem_st8(lane() + L + j, l);
        }
        gf_tmem_wait_st();
    }
    static __device__ __forceinline__ void put(unsigned at, float x, unsigned loAt) {
        const float h = gf_tf32(x);
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(at), "f"(h) : "memory");
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + loAt), "f"(x - h) : "memory");
    }
    __device__ __forceinline__ void column(int i, float x, float e) {
        const unsigned sw = (unsigned)(i & 7) << 4;
        put((store ^ sw) + (unsigned)(rowOf(0, i) - rowOf(0, 0)) * 128u, x, ABYTES);
        if(WT && i < 2 * NA)
            put((storeB ^ sw) + (unsigned)i * 128u, x * e, BBYTES);
    }
    // Shared-memory matrix descriptor: start >> 4 (bits 0-13), leading offset (unused in this layout: 1), stride
    // between 8-row groups 1024 >> 4 (bits 32-45), version 1 (bits 46-47), 128-byte swizzle (2 in bits 61-63).  The low word
    // of base; an operand at an offset adds the offset >> 4 to it.
    __device__ __forceinline__ unsigned desc() const { return ((base >> 4) & 0x3FFFu) | (1u << 16); }
    static __device__ __forceinline__ void mma(unsigned d, unsigned a, unsigned b, unsigned accumulate) {
        asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %4, 0;\n\tmov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %5};\n\t"
                     "tcgen05.mma.cta_group::1.kind::tf32 [%0], da, db, %3, p;\n\t}\n" ::"r"(d), "r"(a), "r"(b),
                     "r"(IDESC), "r"(accumulate), "r"(64u | (1u << 14) | (2u << 29)) : "memory");
    }
    // Tile u: this thread's point (values A, derivatives dA, efficiency e; zeros outside the set).  False on every
    // thread when the wait for the previous tile's MMAs ran out in any.
    __device__ __forceinline__ bool tile(int u, const float2 *A, const float2 *dA, float e) {
        bool ok = true;
        if(u > 0)
            ok = wait(u - 1);
        if(ok) { // the MMAs of the tile before have read its operands
#pragma unroll
            for(int c = 0; c < NC; ++c) {
                const float2 x = c < NA ? A[c < NA ? c : 0] : dA[c < NA ? 0 : c - NA];
                column(2 * c, x.x, e);
                column(2 * c + 1, x.y, e);
            }
            if(u > 0) // after the stores: the drain's registers do not compete with the columns'
                drain();
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        gf_tc_before();
        if(__syncthreads_or(!ok))
            return false;
        if(threadIdx.x < 32 * KB && gf_elect()) {
            gf_tc_after();
            const int b = KB == 1 ? 0 : (int)(threadIdx.x >> 5);
            constexpr unsigned AL = ABYTES >> 4, BH = WT ? 2 * AL : 0u, BL = WT ? BH + (BBYTES >> 4) : AL;
            const unsigned oa = desc() + b * 1024u, ob = desc() + (WT ? b * N * 8u : b * 1024u), d = tmem + (unsigned)(b * N);
#pragma unroll
            for(int k = 0; k < 4; ++k) { // 8 points: 32 bytes of every 128-byte row
                mma(d, oa + AL + 2 * k, ob + BL + 2 * k, k > 0);
                mma(d, oa + 2 * k, ob + BL + 2 * k, 1u);
                mma(d, oa + AL + 2 * k, ob + BH + 2 * k, 1u);
            }
#pragma unroll
            for(int k = 0; k < 4; ++k)
                mma(d, oa + 2 * k, ob + BH + 2 * k, 1u);
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(gf_s32(&sh->mbar)) : "memory");
        }
        last = u;
        return true;
    }
    // Ends the CTA's pass: its sums over the slices, in FP64, to out[entry * gridDim.x + blockIdx.x]; frees the tensor
    // memory.  After a wait that ran out (here or in tile) GF_GRAM_STOPPED in their place.
    __device__ __forceinline__ void end(bool ok, double *out) {
        if(ok && last >= 0) {
            ok = wait(last);
            if(ok)
                drain();
        }
        if(__syncthreads_or(!ok)) {
            // the last committed MMAs must have ended before the tensor memory goes away (2 s, whatever the limit)
            if(last >= 0)
                gf_mbar_wait(&sh->mbar, (unsigned)(last & 1), 2000000000ull);
            ok = false;
        }
        double *red = reinterpret_cast<double *>(ops);
        if(ok)
#pragma unroll
            for(int j = 0; j < WN; j += 8) {
                float h[8], l[8];
                gf_tmem_ld8(lane() + H + j, h);
                gf_tmem_ld8(lane() + L + j, l);
                gf_tmem_wait_ld();
                gf_tmem_got(h);
                gf_tmem_got(l);
#pragma unroll
                for(int i = 0; i < 8; ++i)
                    red[threadIdx.x * WN + j + i] = (double)h[i] + (double)l[i];
            }
        gf_tc_before();
        __syncthreads();
        gf_tc_after();
        if(threadIdx.x < 32)
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS) : "memory");
        if(!ok) {
            for(int q = threadIdx.x; q < 4 * NC * NA; q += 128)
                reinterpret_cast<unsigned long long *>(out)[(i64)q * gridDim.x + blockIdx.x] = GF_GRAM_STOPPED;
            return;
        }
        for(int q = threadIdx.x; q < 4 * NC * NA; q += 128) {
            const int i = q / (2 * NA), j = q % (2 * NA);
            double t = 0.0;
            for(int s = 0; s < S; ++s)
                t += red[rowOf(s, i) * WN + j];
            out[(i64)q * gridDim.x + blockIdx.x] = t;
        }
    }
};

// entry blockIdx.x of every node's G: the sum over the CTAs' partials, FP64; GF_GRAM_STOPPED when a CTA stopped
extern "C" __global__ void __launch_bounds__(128) gf_ampng_sum(const GfArgs a) {
    __shared__ double red[4];
    double s = 0.0;
    bool stopped = false;
    gf_pdl_wait();
    for(int b = threadIdx.x; b < a.gram_ctas; b += 128) {
        const double v = a.gpart[(i64)blockIdx.x * a.gram_ctas + b];
        stopped |= (unsigned long long)__double_as_longlong(v) == GF_GRAM_STOPPED;
        s += v;
    }
#pragma unroll
    for(int o = 16; o > 0; o >>= 1)
        s += __shfl_xor_sync(0xffffffffu, s, o);
    if((threadIdx.x & 31) == 0)
        red[threadIdx.x >> 5] = s;
    stopped = __syncthreads_or(stopped);
    if(threadIdx.x == 0) {
        if(stopped)
            reinterpret_cast<unsigned long long *>(a.gout)[blockIdx.x] = GF_GRAM_STOPPED;
        else
            a.gout[blockIdx.x] = (red[0] + red[1]) + (red[2] + red[3]);
    }
}
)CUDA";

} // namespace gf
