// ---------------------------------------------------------------------------
// fa_steps.cu -- the reference's FA2 build-order steps on warp primitives.
//
//   step 0  fa_naive  research/flash-attention-mi300x/fa_naive.hip:72-212
//           one wave per query row, portable shfl_down softmax reductions
//   step 1  fa_dpp    research/flash-attention-mi300x/fa_dpp.hip:52-167
//           the same with wave::dpp::reduce_max_bcast / reduce_sum_bcast
//   step 2  fa_dme    research/flash-attention-mi300x/fa_dme.hip:74-221
//           step 1 + K/V tiles double-buffered by asynchronous copies (cp.async)
//   (step 3, fa_mfma2, is the tcgen05 kernel in prefill.cu)
// and, with fp32 I/O, the reference's fp32 kernels
//   research/flash-attention-mi300x/kernels/fa_naive.hip:118-278
//   research/flash-attention-mi300x/kernels/fa_dpp.hip:167-313
// whose launch takes (seq_len, n_heads, scale).
//
// Tiling is the reference's: Br = 16 query rows per CTA (four or two per warp),
// Bc = 64 keys per tile.  A 64-key score row is held by ONE 32-lane warp as an
// adjacent pair per lane (keys 2l, 2l+1), which is exactly the shape the pair
// overloads of wave64.cuh reduce; O stays in registers (D/32 dims per lane)
// instead of the reference's LDS accumulator.
// These kernels exist for parity with the reference's steps and to exercise the
// primitives in a simple setting; at the reference's config
// (0.54 GFLOP, 4 MiB) shared memory bounds them (below).
// ---------------------------------------------------------------------------
#include "common.cuh"
#include "attn_common.cuh"
#include "dme/dme_tma.cuh"
#include "wave_primitives/wave64.cuh"

namespace b200p {
int prefill_dispatch(const void* Q, const void* K, const void* V, void* O, const b200p_prefill_cfg* c, int dtype,
                     float* debug_s, cudaStream_t st);
namespace {

constexpr int kBr = 16, kBc = 64;

// The reference's portable reduction: v op= shfl_down(v, o), then broadcast lane 0
// (fa_naive.hip:48-58), on a pair per lane.
template <typename Op>
__device__ __forceinline__ float portable_reduce_bcast(float a, float b, Op op) {
    float v = op(a, b);
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_down_sync(0xffffffffu, v, o));
    return __shfl_sync(0xffffffffu, v, 0);
}

template <typename T> __device__ __forceinline__ float exp_for(float x);
template <> __device__ __forceinline__ float exp_for<float>(float x)         { return expf(x); }
template <> __device__ __forceinline__ float exp_for<__half>(float x)        { return __expf(x); }
template <> __device__ __forceinline__ float exp_for<__nv_bfloat16>(float x) { return __expf(x); }

// What bounds this kernel is shared memory: a warp reads the whole K and V tile for its rows, and q and the weights as broadcasts.
// Two 16-byte reads of K per lane (8 wavefronts) serve all rows of the warp, each row's q one more: 32 FMAs a lane cost 12 wavefronts
// with four rows, 20 with two and 36 with one.  So that there are still eight warps for 16 rows, they are two groups
// that take every other tile; the second group's maxima, sums and O join the first's at the end.  (fp32 heads of 128: one group of two
// rows a warp, two tiles would leave no second CTA.)  Every lane reads its own two key rows at the same 16-byte chunk, so q is a
// broadcast; the keys lie 16 bytes further apart than their size, odd keys behind the even ones, and the eight lanes of a
// shared-memory phase hit eight different bank groups.  Against one group of two rows a warp, graph replays, step 1 / step 2: 8 heads of
// 64, 512 keys, fp32 37.9 / 34.3 -> 30.6 / 29.1 us, fp16 30.7 / 30.5 -> 25.7 / 24.6; 24 heads, 1024 keys, fp32 353 / 327 -> 306 / 287;
// fp16, heads of 128, 497 / 505 -> 431 / 408.  Counted for the first of these, fp32, step 2: 6.6 -> 4.6 million wavefronts.
// Lengths need not be multiples of the tiles: keys past the end get no weight, rows past the end are not stored.
constexpr int kStepWarps = 8, kStepThreads = kStepWarps * 32;
template <typename T, int D> struct StepTile {
    static constexpr int MAX_G = D * int(sizeof(T)) <= 256 ? 2 : 1;       // groups of warps (below) whose tiles fit an SM
    static constexpr int ROW = D * int(sizeof(T));                         // bytes of a key
    static constexpr int KROW = ROW + 16;                                  // between two slots of K
    static constexpr int K_BYTES = kBc * KROW, V_BYTES = kBc * ROW;
};

// G groups of warps, KB and VB buffers of their tiles of K and V (step 2: 2 and 2, 2 and 1, or 1 and 1; the others: 1 and 1)
// CTAs an SM the registers are bound for: fp32 heads of 128, steps 1 and 2, 8 heads, 512 keys, 64.7 and 60.6 us with 2, 62.8 and 58.9 with
// 1.  (Unbound, with 60 registers, they take 2 to 3 % less where all rounds of CTAs are full, and up to a quarter more where the last one
// is not: 8 heads, 512 / 831 keys, step 1 63.0 / 195 against 64.7 / 160 us.)
template <typename T, int D, int STEP, int G, int KB, int VB>
__global__ void __launch_bounds__(kStepThreads, D * sizeof(T) > 256 && STEP != 0 ? 1 : 2)
fa_step_kernel(const T* __restrict__ Q, const T* __restrict__ K, const T* __restrict__ V, T* __restrict__ O,
               int seq_q, int seq_k, int heads, float scale, float m_first) {
    using Sh = StepTile<T, D>;
    constexpr int DPL = D / 32;                           // output dims per lane
    constexpr int R = 2 * G, WG = kStepWarps / G;                         // rows per warp, warps of a group
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char* Kt = smem;                                              // [KB][G][kBc slots][KROW]: key k in slot (k % 2) * 32 + k / 2
    unsigned char* Vt = smem + KB * G * Sh::K_BYTES;                       // [VB][G][kBc][D]
    float* prow = reinterpret_cast<float*>(Vt + VB * G * Sh::V_BYTES);     // [G][Br][Bc]
    float* qs = prow + G * kBr * kBc;                                      // [Br][D]

    // blockIdx.x = batch * heads * (seq_q/Br) + head * (seq_q/Br) + qblk   (fa_naive.hip:70-71)
    const int qblocks = (seq_q + kBr - 1) / kBr;
    const int qblk = blockIdx.x % qblocks;
    const int bh = blockIdx.x / qblocks;                                   // batch * heads + head
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int wrow = warp % WG * R, grp = warp / WG;                       // this warp's first row of the block, its group
    const int row0 = qblk * kBr + wrow;                                    // this warp's first query row
    const T* Kb = K + size_t(bh) * seq_k * D;
    const T* Vb = V + size_t(bh) * seq_k * D;
    const int ntiles = (seq_k + kBc - 1) / kBc;

    float* q = qs + wrow * D;
    #pragma unroll
    for (int r = grp; r < R; r += G)                                       // (read behind the first tile's barrier)
        for (int d = lane; d < D; d += 32) q[r * D + d] = row0 + r < seq_q ? to_float(Q[(size_t(bh) * seq_q + row0 + r) * D + d]) : 0.f;
    // K, V or both of tiles j * G .. into their buffers, 16 bytes per thread per step: asynchronous copies (step 2), or through registers
    auto copy = [&](int j, bool of_k, bool of_v) {
        constexpr int CPR = Sh::ROW / 16;                                 // chunks per key
        #pragma unroll
        for (int t = 0; t < G; ++t) {
            const int k0 = (j * G + t) * kBc, n = min(kBc, seq_k - k0);
            const uint4* ks = reinterpret_cast<const uint4*>(Kb + size_t(k0) * D);
            const uint4* vs = reinterpret_cast<const uint4*>(Vb + size_t(k0) * D);
            unsigned char* kd = Kt + (j % KB * G + t) * Sh::K_BYTES;
            unsigned char* vd = Vt + (j % VB * G + t) * Sh::V_BYTES;
            for (int i = threadIdx.x; i < n * CPR; i += kStepThreads) {
                const int k = i / CPR, c = i % CPR;
                unsigned char* kslot = kd + ((k & 1) * 32 + (k >> 1)) * Sh::KROW + c * 16;
                if (STEP == 2) {
                    if (of_k) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dme::smem_addr(kslot)), "l"(ks + i) : "memory");
                    if (of_v) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dme::smem_addr(vd + i * 16)), "l"(vs + i) : "memory");
                } else {
                    *reinterpret_cast<uint4*>(kslot) = ks[i];
                    reinterpret_cast<uint4*>(vd)[i] = vs[i];
                }
            }
        }
        if (STEP == 2) asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (KB == 2) copy(0, true, VB == 2);

    float* const pw = prow + (grp * kBr + wrow) * kBc;                      // this warp's weights
    float m[R], l[R], o[R][DPL];
    #pragma unroll
    for (int r = 0; r < R; ++r) {
        m[r] = m_first; l[r] = 0.f;
        #pragma unroll
        for (int i = 0; i < DPL; ++i) o[r][i] = 0.f;
    }

    const int steps = (ntiles + G - 1) / G;
    for (int j = 0; j < steps; ++j) {
        const int buf = KB == 2 ? (j & 1) : 0, live = min(kBc, seq_k - (j * G + grp) * kBc);
        const unsigned char* Kc = Kt + (buf * G + grp) * Sh::K_BYTES;
        const unsigned char* Vc = Vt + (j % VB * G + grp) * Sh::V_BYTES;
        // no weight times whatever was there must be nothing
        auto clear_tail = [&] {
            if (j + 1 < steps || seq_k % kBc == 0) return;
            uint4* Vl = reinterpret_cast<uint4*>(Vt + (j % VB * G + (ntiles - 1) % G) * Sh::V_BYTES);
            for (int i = seq_k % kBc * (Sh::ROW / 16) + threadIdx.x; i < kBc * (Sh::ROW / 16); i += kStepThreads) Vl[i] = make_uint4(0u, 0u, 0u, 0u);
        };
        if (KB == 2 && VB == 1) {                                          // V travels under the scores, the next K under the whole step
            copy(j, false, true);
            if (j + 1 < steps) { copy(j + 1, true, false); asm volatile("cp.async.wait_group 2;" ::: "memory"); }
            else asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else if (KB == 2) {                                              // prefetch the next tiles, wait for these
            if (j + 1 < steps) { copy(j + 1, true, true); asm volatile("cp.async.wait_group 1;" ::: "memory"); }
            else asm volatile("cp.async.wait_group 0;" ::: "memory");
            clear_tail();
        } else {
            copy(j, true, true);
            if (STEP == 2) asm volatile("cp.async.wait_group 0;" ::: "memory");
            clear_tail();
        }
        __syncthreads();
        if (G == 1 || live > 0) {                                          // (the last step may have no tile for this group)
        // S[row][2l], S[row][2l+1]
        float s0[R], s1[R];
        #pragma unroll
        for (int r = 0; r < R; ++r) s0[r] = s1[r] = 0.f;
        {
            constexpr int EPC = 16 / int(sizeof(T)), NCH = D / EPC;       // elements per chunk, chunks per row
            const uint4* kr0 = reinterpret_cast<const uint4*>(Kc + lane * Sh::KROW);
            const uint4* kr1 = reinterpret_cast<const uint4*>(Kc + (32 + lane) * Sh::KROW);
            #pragma unroll 4
            for (int c = 0; c < NCH; ++c) {
                const uint4 ka = kr0[c], kb = kr1[c];
                const T* ea = reinterpret_cast<const T*>(&ka);
                const T* eb = reinterpret_cast<const T*>(&kb);
                #pragma unroll
                for (int r = 0; r < R; ++r) {
                    float qv[EPC];
                    #pragma unroll
                    for (int e = 0; e < EPC; e += 4) *reinterpret_cast<float4*>(&qv[e]) = *reinterpret_cast<const float4*>(q + r * D + c * EPC + e);
                    #pragma unroll
                    for (int e = 0; e < EPC; ++e) { s0[r] = fmaf(qv[e], to_float(ea[e]), s0[r]); s1[r] = fmaf(qv[e], to_float(eb[e]), s1[r]); }
                }
            }
        }
        // online softmax (cdna3-prims/examples/fused_softmax.hpp:38-48)
        #pragma unroll
        for (int r = 0; r < R; ++r) {
            constexpr float kLowest = -3.402823466e+38f;
            s0[r] = 2 * lane < live ? s0[r] * scale : kLowest;
            s1[r] = 2 * lane + 1 < live ? s1[r] * scale : kLowest;
            const float rmax = STEP == 0 ? portable_reduce_bcast(s0[r], s1[r], wave::MaxOp{}) : wave::dpp::reduce_max_bcast(s0[r], s1[r]);
            const float m_new = fmaxf(m[r], rmax);
            const float p0 = 2 * lane < live ? exp_for<T>(s0[r] - m_new) : 0.f, p1 = 2 * lane + 1 < live ? exp_for<T>(s1[r] - m_new) : 0.f;
            const float rsum = STEP == 0 ? portable_reduce_bcast(p0, p1, wave::SumOp{}) : wave::dpp::reduce_sum_bcast(p0, p1);
            const float resc = exp_for<T>(m[r] - m_new);
            l[r] = resc * l[r] + rsum;
            m[r] = m_new;
            #pragma unroll
            for (int i = 0; i < DPL; ++i) o[r][i] *= resc;
            *reinterpret_cast<float2*>(&pw[r * kBc + 2 * lane]) = make_float2(p0, p1);
        }
        __syncwarp();
        }
        if (KB == 2 && VB == 1) {
            if (j + 1 < steps) asm volatile("cp.async.wait_group 1;" ::: "memory");
            else asm volatile("cp.async.wait_group 0;" ::: "memory");
            clear_tail();
            __syncthreads();
        }
        if (G == 1 || live > 0) {
        // O[row][d] += sum_k P[row][k] * V[k][d]
        #pragma unroll 2
        for (int k = 0; k < kBc; k += 4) {
            float4 p4[R];
            #pragma unroll
            for (int r = 0; r < R; ++r) p4[r] = *reinterpret_cast<const float4*>(&pw[r * kBc + k]);      // broadcast reads
            #pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                float v[DPL];
                #pragma unroll
                for (int i = 0; i < DPL; ++i) v[i] = to_float(reinterpret_cast<const T*>(Vc)[(k + kk) * D + lane * DPL + i]);
                #pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float pk = kk == 0 ? p4[r].x : kk == 1 ? p4[r].y : kk == 2 ? p4[r].z : p4[r].w;
                    #pragma unroll
                    for (int i = 0; i < DPL; ++i) o[r][i] = fmaf(pk, v[i], o[r][i]);
                }
            }
        }
        }
        __syncthreads();                                  // tile buffers and prow are reused next iteration
    }
    if (G == 2) {                                         // the second group's part of the rows joins the first's
        float* part = reinterpret_cast<float*>(Kt) + (warp % WG) * R * (D + 2);       // [R][D] sums, [R] m, [R] l
        static_assert(WG * R * (D + 2) * int(sizeof(float)) <= Sh::K_BYTES);
        if (grp == 1) {
            #pragma unroll
            for (int r = 0; r < R; ++r) {
                #pragma unroll
                for (int i = 0; i < DPL; ++i) part[r * D + lane * DPL + i] = o[r][i];
                if (lane == 0) { part[R * D + r] = m[r]; part[R * D + R + r] = l[r]; }
            }
        }
        __syncthreads();
        if (grp == 1) return;
        #pragma unroll
        for (int r = 0; r < R; ++r) {
            const float mo = part[R * D + r], m_new = fmaxf(m[r], mo), a = exp_for<T>(m[r] - m_new), b = exp_for<T>(mo - m_new);
            l[r] = a * l[r] + b * part[R * D + R + r];
            #pragma unroll
            for (int i = 0; i < DPL; ++i) o[r][i] = a * o[r][i] + b * part[r * D + lane * DPL + i];
        }
    }
    #pragma unroll
    for (int r = 0; r < R; ++r) {
        const float inv = l[r] > 0.f ? 1.f / l[r] : 0.f;  // kernels/fa_naive.hip: l_inv = l > 0 ? 1/l : 0
        if (row0 + r < seq_q) {
            #pragma unroll
            for (int i = 0; i < DPL; ++i) O[(size_t(bh) * seq_q + row0 + r) * D + lane * DPL + i] = from_float<T>(o[r][i] * inv);
        }
    }
}

// ---------------------------------------------------------------------------
// The reference's fp32-I/O kernels, one query row per block (Br = 1):
//   research/flash-attention-mi300x/kernels/fa_naive.hip:118-278   (DPP = false)
//   research/flash-attention-mi300x/kernels/fa_dpp.hip:96-155,167-313 (DPP = true)
// Bc keys per tile are spread over Bc/64 "waves"; here a wave is one 32-lane warp
// holding the 64 scores as an adjacent pair per lane.  Row max and row sum are the
// reference's two-phase reduction (block_reduce_max_sum): inside the wave with the
// pair primitives (shfl_down order for the naive kernel), across the waves through
// 2 * waves floats of shared memory.  Keys past seq_len are padded with the lowest
// float and contribute p = 0 (kernels/fa_naive.hip:158-169,233); any seq_len works.
// O[row] = sum_k p_k V[k] / l with l_inv = l > 0 ? 1/l : 0.
// ---------------------------------------------------------------------------
template <int BC, int D, bool DPP>
__global__ void __launch_bounds__(BC / 2)
fa_rows_f32_kernel(const float* __restrict__ Q, const float* __restrict__ K, const float* __restrict__ V,
                   float* __restrict__ O, int seq_len, int n_heads, float scale) {
    constexpr int WAVES = BC / 64, THREADS = BC / 2;
    constexpr float kLowest = -3.402823466e+38f;
    __shared__ __align__(16) float q_s[D];
    __shared__ float p_s[BC];
    __shared__ float red[2 * WAVES];
    const int tid = threadIdx.x, wave_i = tid / 32, lane = tid % 32;
    const int row = blockIdx.x, bh = blockIdx.y;               // bh = batch * n_heads + head
    const size_t base = size_t(bh) * seq_len * D;
    for (int d = tid; d < D; d += THREADS) q_s[d] = Q[base + size_t(row) * D + d];
    __syncthreads();

    float m = kLowest, l = 0.f;
    constexpr int DPT = (D + THREADS - 1) / THREADS;           // output dims per thread: d = tid + i * THREADS
    float o[DPT];
    #pragma unroll
    for (int i = 0; i < DPT; ++i) o[i] = 0.f;

    const int tiles = (seq_len + BC - 1) / BC;
    for (int j = 0; j < tiles; ++j) {
        const int kv0 = j * BC;
        const int k0 = kv0 + wave_i * 64 + 2 * lane, k1 = k0 + 1;
        float s0 = kLowest, s1 = kLowest;
        if (k0 < seq_len) {
            const float4* kr = reinterpret_cast<const float4*>(K + base + size_t(k0) * D);
            float a = 0.f;
            #pragma unroll 4
            for (int d4 = 0; d4 < D / 4; ++d4) {
                const float4 kv = kr[d4]; const float4 qv = *reinterpret_cast<const float4*>(&q_s[4 * d4]);
                a = fmaf(qv.x, kv.x, a); a = fmaf(qv.y, kv.y, a); a = fmaf(qv.z, kv.z, a); a = fmaf(qv.w, kv.w, a);
            }
            s0 = a * scale;
        }
        if (k1 < seq_len) {
            const float4* kr = reinterpret_cast<const float4*>(K + base + size_t(k1) * D);
            float a = 0.f;
            #pragma unroll 4
            for (int d4 = 0; d4 < D / 4; ++d4) {
                const float4 kv = kr[d4]; const float4 qv = *reinterpret_cast<const float4*>(&q_s[4 * d4]);
                a = fmaf(qv.x, kv.x, a); a = fmaf(qv.y, kv.y, a); a = fmaf(qv.z, kv.z, a); a = fmaf(qv.w, kv.w, a);
            }
            s1 = a * scale;
        }
        // phase 1: inside the wave; phase 2: across the waves of the block
        float tmax = DPP ? wave::dpp::reduce_max_bcast(s0, s1) : portable_reduce_bcast(s0, s1, wave::MaxOp{});
        if (WAVES > 1) {
            if (lane == 0) red[wave_i] = tmax;
            __syncthreads();
            tmax = red[0];
            #pragma unroll
            for (int w = 1; w < WAVES; ++w) tmax = tmax > red[w] ? tmax : red[w];
        }
        const float m_new = fmaxf(m, tmax);                    // running max (fused_softmax.hpp:38-48)
        const float p0 = k0 < seq_len ? expf(s0 - m_new) : 0.f;
        const float p1 = k1 < seq_len ? expf(s1 - m_new) : 0.f;
        float tsum = DPP ? wave::dpp::reduce_sum_bcast(p0, p1) : portable_reduce_bcast(p0, p1, wave::SumOp{});
        if (WAVES > 1) {
            if (lane == 0) red[WAVES + wave_i] = tsum;
            __syncthreads();
            tsum = red[WAVES];
            #pragma unroll
            for (int w = 1; w < WAVES; ++w) tsum += red[WAVES + w];
        }
        const float alpha = expf(m - m_new);
        m = m_new;
        l = alpha * l + tsum;
        p_s[wave_i * 64 + 2 * lane] = p0;
        p_s[wave_i * 64 + 2 * lane + 1] = p1;
        __syncthreads();
        const int live = min(BC, seq_len - kv0);
        #pragma unroll
        for (int i = 0; i < DPT; ++i) {
            const int d = tid + i * THREADS;
            if (d < D) {
                float acc = o[i] * alpha;
                const float* vcol = V + base + size_t(kv0) * D + d;
                #pragma unroll 4
                for (int k = 0; k < live; ++k) acc = fmaf(p_s[k], vcol[size_t(k) * D], acc);
                o[i] = acc;
            }
        }
        __syncthreads();                                       // p_s and red are rewritten by the next tile
    }
    const float l_inv = l > 0.f ? 1.f / l : 0.f;
    #pragma unroll
    for (int i = 0; i < DPT; ++i) {
        const int d = tid + i * THREADS;
        if (d < D) O[base + size_t(row) * D + d] = o[i] * l_inv;
    }
}

template <int BC, int D>
int launch_rows(bool dpp, const float* Q, const float* K, const float* V, float* O, int batch, int heads, int seq_len,
                float scale, cudaStream_t st) {
    const dim3 grid(unsigned(seq_len), unsigned(batch) * unsigned(heads));
    if (dpp) fa_rows_f32_kernel<BC, D, true><<<grid, BC / 2, 0, st>>>(Q, K, V, O, seq_len, heads, scale);
    else     fa_rows_f32_kernel<BC, D, false><<<grid, BC / 2, 0, st>>>(Q, K, V, O, seq_len, heads, scale);
    return launched();
}
template <int D>
int launch_rows_bc(int bc, bool dpp, const float* Q, const float* K, const float* V, float* O, int batch, int heads,
                   int seq_len, float scale, cudaStream_t st) {
    switch (bc) {
        case 64:  return launch_rows<64, D>(dpp, Q, K, V, O, batch, heads, seq_len, scale, st);
        case 128: return launch_rows<128, D>(dpp, Q, K, V, O, batch, heads, seq_len, scale, st);
        case 256: return launch_rows<256, D>(dpp, Q, K, V, O, batch, heads, seq_len, scale, st);
    }
    return B200P_E_OP;
}

template <typename T, int D, int STEP>
int launch_step(const void* Q, const void* K, const void* V, void* O, int batch, int heads, int seq_q, int seq_k,
                float scale, float m_first, cudaStream_t st) {
    using Sh = StepTile<T, D>;
    // two groups of warps wherever there are two tiles for them (one tile, 1 head of 64, fp16: 4.4 us with one, 5.2 with two)
    const int G = seq_k > kBc ? Sh::MAX_G : 1;
    const unsigned grid = unsigned(batch) * heads * ((seq_q + kBr - 1) / kBr);
    // Step 2's fp32 tiles with one buffer of V leave room for a second CTA on an SM, if there is one (8 heads of 64, 512 keys: 36.0 us with two
    // buffers, 28.3 with one; of 128: 68.9 and 58.9, but 1 head 35.0 and 36.8; fp16, 8 heads of 128: 47.2 and 50.1).  Two groups' 16-bit tiles of
    // 128 columns leave it with one buffer of either: the second CTA then computes while the first one copies.  fp16, 24 heads of 128, step 2 with one
    // group, with two and two buffers, with two and one: 128 keys 15.3 / 16.5 / 13.5 us, 192 21.5 / 23.2 / 19.0, 512 142 / 137 / 117, 1024 505 / 473 / 408.
    constexpr int MOST = STEP == 2 ? 2 : 1;
    const bool share = STEP == 2 && grid > unsigned(sm_count()), one = share && sizeof(T) == 2 && G * D == 256;
    const int KB = one ? 1 : MOST, VB = one || (share && sizeof(T) == 4) ? 1 : MOST;
    const size_t smem = G * (size_t(KB) * Sh::K_BYTES + size_t(VB) * Sh::V_BYTES) + (G * kBr * kBc + kBr * D) * sizeof(float);
    auto kern = G == 2 ? fa_step_kernel<T, D, STEP, Sh::MAX_G, MOST, MOST> : fa_step_kernel<T, D, STEP, 1, MOST, MOST>;
    if constexpr (sizeof(T) == 4) if (VB < MOST) kern = G == 2 ? fa_step_kernel<T, D, STEP, Sh::MAX_G, MOST, 1> : fa_step_kernel<T, D, STEP, 1, MOST, 1>;
    if constexpr (sizeof(T) == 2 && D == 128) if (KB < MOST) kern = fa_step_kernel<T, D, STEP, 2, 1, 1>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        if (e != cudaSuccess) return int(e);
    }
    kern<<<grid, kStepThreads, smem, st>>>(static_cast<const T*>(Q), static_cast<const T*>(K), static_cast<const T*>(V),
                                       static_cast<T*>(O), seq_q, seq_k, heads, scale, m_first);
    return launched();
}
template <typename T, int D>
int launch_step_s(int step, const void* Q, const void* K, const void* V, void* O, int batch, int heads, int seq_q,
                  int seq_k, float scale, float m_first, cudaStream_t st) {
    switch (step) {
        case 0: return launch_step<T, D, 0>(Q, K, V, O, batch, heads, seq_q, seq_k, scale, m_first, st);
        case 1: return launch_step<T, D, 1>(Q, K, V, O, batch, heads, seq_q, seq_k, scale, m_first, st);
        case 2: return launch_step<T, D, 2>(Q, K, V, O, batch, heads, seq_q, seq_k, scale, m_first, st);
    }
    return B200P_E_OP;
}
template <typename T>
int launch_step_d(int step, int D, const void* Q, const void* K, const void* V, void* O, int batch, int heads,
                  int seq_q, int seq_k, float scale, float m_first, cudaStream_t st) {
    return D == 64 ? launch_step_s<T, 64>(step, Q, K, V, O, batch, heads, seq_q, seq_k, scale, m_first, st)
                   : launch_step_s<T, 128>(step, Q, K, V, O, batch, heads, seq_q, seq_k, scale, m_first, st);
}

} // namespace
} // namespace b200p

using namespace b200p;

extern "C" int b200p_fa_rows_f32(int variant, int bc, const float* Q, const float* K, const float* V, float* O,
                                 int batch, int heads, int seq_len, int D, float scale, b200p_stream_t stream) {
    if (variant != 0 && variant != 1) return B200P_E_OP;
    if (bc != 64 && bc != 128 && bc != 256) return B200P_E_OP;
    if (D != 64 && D != 128) return B200P_E_DIM;
    if (batch <= 0 || heads <= 0 || seq_len <= 0) return B200P_E_LENGTH;
    if ((long long)batch * heads > 65535) return B200P_E_RANGE;
    if (!Q || !K || !V || !O) return B200P_E_NULL;
    if (!aligned(Q, 16) || !aligned(K, 16) || !aligned(V, 16) || !aligned(O, 16)) return B200P_E_ALIGN;
    if (sm_count() <= 0) return B200P_E_NO_DEVICE;
    if (scale == 0.f) scale = 1.f / sqrtf(float(D));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return D == 64 ? launch_rows_bc<64>(bc, variant == 1, Q, K, V, O, batch, heads, seq_len, scale, st)
                   : launch_rows_bc<128>(bc, variant == 1, Q, K, V, O, batch, heads, seq_len, scale, st);
}

extern "C" int b200p_fa_step(int step, int dtype, const void* Q, const void* K, const void* V, void* O,
                             int batch, int heads, int seq_q, int seq_k, int D, float scale, b200p_stream_t stream) {
    if (step < 0 || step > 3) return B200P_E_OP;
    if (dtype != B200P_F16 && dtype != B200P_BF16 && dtype != B200P_F32) return B200P_E_DTYPE;
    if (D != 64 && D != 128) return B200P_E_DIM;
    if (batch <= 0 || heads <= 0 || seq_q <= 0 || seq_k <= 0) return B200P_E_LENGTH;
    if (!Q || !K || !V || !O) return B200P_E_NULL;
    if (!aligned(Q, 16) || !aligned(K, 16) || !aligned(V, 16) || !aligned(O, 16)) return B200P_E_ALIGN;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (step == 3) {
        // the tensor-core step: 16-bit operands, fixed scale 1/sqrt(D) like fa_mfma2.hip
        if (dtype == B200P_F32) return B200P_E_DTYPE;
        if (scale != 0.f && fabsf(scale * sqrtf(float(D)) - 1.f) > 1e-6f) return B200P_E_OP;
        b200p_prefill_cfg c{D, seq_q, seq_k, heads, heads, batch, 0};
        return prefill_dispatch(Q, K, V, O, &c, dtype, nullptr, st);
    }
    if (sm_count() <= 0) return B200P_E_NO_DEVICE;
    if (scale == 0.f) scale = 1.f / sqrtf(float(D));
    float m_first = -1e38f;                                // the reference's initial running max
    if (seq_q % kBr != 0 || seq_k % kBc != 0) {
        // Lengths off the Br = 16 / Bc = 64 tiling: fp32 I/O takes any seq_len like the reference's fp32 kernels, whose running
        // max starts at the lowest float (kernels/fa_naive.hip:158-169); the 16-bit steps keep the reference's tiling.
        if (dtype != B200P_F32 || seq_q != seq_k) return B200P_E_LENGTH;
        if ((long long)batch * heads > 65535) return B200P_E_RANGE;      // as in b200p_fa_rows_f32, the other entry for such lengths
        m_first = -3.402823466e+38f;
    }
    switch (dtype) {
        case B200P_F16:  return launch_step_d<__half>(step, D, Q, K, V, O, batch, heads, seq_q, seq_k, scale, m_first, st);
        case B200P_BF16: return launch_step_d<__nv_bfloat16>(step, D, Q, K, V, O, batch, heads, seq_q, seq_k, scale, m_first, st);
        default:         return launch_step_d<float>(step, D, Q, K, V, O, batch, heads, seq_q, seq_k, scale, m_first, st);
    }
}
