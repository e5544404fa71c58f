// ---------------------------------------------------------------------------
// skinny_tc.cuh -- Y[M,N] = X[M,K] . W[N,K]^T for up to 16 rows of X, with K split over a thread-block cluster and
// the products on tcgen05.
//
// skinny_gemm.cuh's kernels keep ALL of X in every CTA: 16 rows of 5632 columns are 180 KB, which leaves no room for
// weight stages; 8 rows of 14336 do not fit at all, and with 16 rows the norm prologue of every CTA reads the whole
// residual stream.  Here a cluster of CS CTAs owns 128 rows of W at a time and CTA r of it owns the r-th slice of K:
//
//  * each CTA holds X[:, slice] only, as 64-column blocks in the 128-byte swizzle the tensor cores read.  Plain 16-bit
//    rows are brought by TMA; a norm prologue reads the slice of the residual stream and the CTAs exchange their
//    sums of squares through distributed shared memory (st.async, completion on the receiver's mbarrier);
//  * a producer thread streams W (128 rows x 64 columns = 16 KB a stage, TMA tensor maps) as far ahead as the ring
//    allows, from before the dependency wait on; one thread issues tcgen05.mma with W as A (M = 128) and X as B
//    (N = 8 or 16), so no register and no warp touches the weights.  (An MMA takes about 40 cycles for any N up to 64,
//    with 64 rows of W as with 128: tiles of 64 rows made the issue of the MMAs slower than HBM.);
//  * two MMAs (32 columns of K) share an accumulator; the workers add the accumulators in fp32 registers, rounded to
//    nearest.  An MMA that accumulates truncates: n of them in a row are off by about 2e-8 n on products of one sign, all
//    downwards, and one accumulator for a whole slice made the outputs up to 25 times less exact than skinny_gemm.cuh's
//    kernels, whose chains are K / 512 long (relative error over normal inputs, 16 rows: N = 32000, K = 2048 9.4e-8 with those
//    kernels, 2.1e-6 with one accumulator a slice, 9.5e-8 now; 4096 x 4096 4.7e-7, 1.0e-6, 8.7e-8; 2048 x 5632 6.6e-7, 9.1e-7,
//    9.2e-8).  One MMA per accumulator is 3 % closer still and 4 to 12 % slower (the workers then read as many bytes of
//    tensor memory as the MMAs read of W: head of 32000 x 4096, 16 rows, 60.2 against 53.9 us; 51.7 with one accumulator a slice);
//  * the partial accumulators are pushed to the CTA of the cluster that owns the outputs (64 / CS row pairs each),
//    again with st.async; the owner adds the CS parts in slice order (the result does not depend on timing) and runs
//    the epilogue.  Accumulators in tensor memory are a ring of kStcSlots blocks and the inboxes are double-buffered: the
//    products of the next tile begin under the exchange of this one.
// What bounds it: the stream of W (HBM), and for one or two tiles per cluster the chain dependency wait -> X -> last
// stage's products -> exchange -> epilogue.  The shared memory is kept below half an SM's where the ring allows, so that the
// next kernel's CTAs are resident and fetch their first stages under this one (prompt and tokens of 8 layers of width 2048, 16
// sequences: 15.6 -> 14.8 ms).
//
// An inbox buffer is written again only after its owner has read it: a CTA pushes tile i+2 after its own inbox of
// tile i+1 is complete, which holds parts that the owner pushed after all its warps had read tile i (worker barrier).
// Waits are bounded.  A wait that gives up raises the abort word, and the thread goes on without waiting, so every
// thread reaches the worker barriers and the cluster barrier at the end.  Where every wait succeeded nobody leaves while
// a peer may still write to its shared memory: each st.async was waited for by its receiver.  After a wait that gave up,
// one that is still on its way is not waited for; the launch has failed by then and says so in the status word.
// ---------------------------------------------------------------------------
#pragma once
#include "skinny_gemm.cuh"
#include "tcgen05.cuh"
#include "tensor_map.cuh"

namespace b200p {

constexpr int kStcRows = 128;                             // rows of W per tile
constexpr int kStcPairs = kStcRows / 2;
constexpr int kStcBlock = 64;                             // columns per swizzled block
constexpr int kStcStageBytes = kStcRows * kStcBlock * 2;  // one block: 16 KB
constexpr int kStcWorkers = 256;
constexpr int kStcThreads = kStcWorkers + 64;             // + producer warp + MMA warp
constexpr int kStcMaxStages = 12;
constexpr int kStcMaxCluster = 8;
constexpr int kStcAccs = 2;                               // accumulators of a block, 16 columns of tensor memory apart
constexpr int kStcSlots = 8;                              // blocks between the MMA warp and the workers
constexpr int kStcSlotCols = kStcAccs * 16;
constexpr int kStcTmemCols = kStcSlots * kStcSlotCols;
// At least a third of an SM's shared memory, so that no more CTAs meet on an SM than its tensor memory serves: a CTA that waited
// for tensor memory could hold up its cluster, and that cluster another one.
constexpr int kStcMinDynamic = 78 * 1024;
static_assert(2 * kStcTmemCols <= 512 && 3 * (kStcMinDynamic + 1024) > 228 * 1024, "two CTAs on an SM, not three");

struct SkinnyTcShape {
    int cluster;          // CTAs sharing K
    int kblocks;          // 64-column blocks of K
    int ntiles;
    int nstages;
    int x_bytes;          // shared memory for X
    int inbox_bytes;      // of one buffer
};
// Floats between two rows of an inbox: 16 bytes more than the row, so that neighbouring rows start on other banks.
__host__ __device__ constexpr int stc_inbox_row(int nb) { return nb + 4; }

__device__ __forceinline__ uint32_t cluster_addr(uint32_t smem, uint32_t cta) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem), "r"(cta));
    return r;
}
// 16 (4) bytes into another CTA's shared memory; that CTA's mbarrier counts them when they have landed.
__device__ __forceinline__ void st_async_v4(uint32_t addr, const uint32_t* v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
                 :: "r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async_f32(uint32_t addr, float v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];"
                 :: "r"(addr), "r"(__float_as_uint(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void stc_worker_barrier() { asm volatile("bar.sync 1, %0;" :: "n"(kStcWorkers) : "memory"); }

template <typename T> struct StcFmt;
template <> struct StcFmt<__half>        { static constexpr int id = 0; };
template <> struct StcFmt<__nv_bfloat16> { static constexpr int id = 1; };

// Pair p (0..63) and half of a tile's accumulator row i, so that what an epilogue needs is in one thread.  EPI_PAIRROT
// pairs rows 8 apart in groups of 16; EPI_ROPE the halves of a head of D (64: two heads a tile); the gated epilogues
// gate row p and up row p, the tile's two boxes; the rest any rows, here 64 apart.
template <int EPI> __device__ __forceinline__ int2 stc_pair(const SkinnyArgs& a, int i) {
    if (EPI == EPI_PAIRROT) return make_int2((i / 16) * 8 + i % 8, (i % 16) / 8);
    if (EPI == EPI_ROPE && a.rope.D == 64) return make_int2((i / 64) * 32 + i % 32, (i % 64) / 32);
    return make_int2(i % kStcPairs, i / kStcPairs);
}
// EPI_ROPE: head (of q, k and v heads in a row) and dimension of a pair.
__device__ __forceinline__ int2 stc_head(const SkinnyRope& r, int tile, int p) {
    return r.D == 64 ? make_int2(tile * 2 + p / 32, p % 32) : make_int2(tile, p);
}

// What the epilogue of (pair p, row m) reads from global memory, asked for before the parts have arrived.
struct StcAhead { float a, b, c, d; };
template <typename T, int EPI>
__device__ __forceinline__ StcAhead stc_fetch(const SkinnyArgs& a, int tile, int p, int m) {
    StcAhead e{0.f, 0.f, 0.f, 0.f};
    if (m >= a.M) return e;
    if (EPI == EPI_ACC32 || EPI == EPI_ADD_FOLD) {
        const int n = tile * kStcRows + p;
        const float* o = static_cast<const float*>(a.out) + size_t(m) * a.ldo;
        if (n < a.N) e.a = o[n];
        if (n + kStcPairs < a.N) e.b = o[n + kStcPairs];
        if (EPI == EPI_ADD_FOLD) {
            const T* w = static_cast<const T*>(a.fold.w);
            if (n < a.N) e.c = to_float(w[n]);
            if (n + kStcPairs < a.N) e.d = to_float(w[n + kStcPairs]);
        }
    } else if (EPI == EPI_ROPE) {
        const SkinnyRope& r = a.rope;
        const int2 hd = stc_head(r, tile, p);
        const int half = r.D / 2, slot = hd.x, d = hd.y;
        if (slot >= r.nQH + 2 * r.nKVH) return e;
        const int pos = r.pos_dev ? min(*r.pos_dev, r.max_seq - 1) : r.pos0;
        if (slot < r.nQH + r.nKVH) { e.a = r.cos_t[size_t(pos) * half + d]; e.b = r.sin_t[size_t(pos) * half + d]; }
        if (r.bias) {
            const T* bias = static_cast<const T*>(r.bias);
            e.c = to_float(bias[slot * r.D + d]); e.d = to_float(bias[slot * r.D + d + half]);
        }
    } else if (EPI == EPI_PAIRROT) {
        const SkinnyPairRot& r = a.pair;
        const int grp = tile * (kStcRows / 16) + p / 8, per_head = r.plain + r.rotated, head = grp * 16 / per_head, j = grp * 16 % per_head;
        if (head < r.heads && j >= r.plain) { const size_t t = pair_angle(r, m, (j - r.plain) / 2 + p % 8); e.a = r.cos_t[t]; e.b = r.sin_t[t]; }
    }
    return e;
}
// The same outputs, rounded at the same places, as skinny_epilogue.  EPI_ADD_FOLD: the sum of squares goes to *sq.
template <typename T, int EPI>
__device__ __forceinline__ void stc_epilogue(const SkinnyArgs& a, int tile, int p, int m, float x0, float x1, const StcAhead& e, float* sq) {
    if (EPI == EPI_ADD_FOLD) *sq = 0.f;
    if (m >= a.M) return;
    if (epi_gated(EPI)) {
        const int n = tile * kStcPairs + p;
        if (n < a.N) static_cast<T*>(a.out)[size_t(m) * a.ldo + n] = from_float<T>(gate_act<EPI>(x0) * x1);
    } else if (EPI == EPI_ROPE) {
        const SkinnyRope& r = a.rope;
        const int2 hd = stc_head(r, tile, p);
        const int half = r.D / 2, slot = hd.x, d = hd.y;
        if (slot >= r.nQH + 2 * r.nKVH) return;
        x0 = to_float(from_float<T>(x0)); x1 = to_float(from_float<T>(x1));      // the projection's 16-bit output
        if (r.bias) { x0 = to_float(from_float<T>(x0 + e.c)); x1 = to_float(from_float<T>(x1 + e.d)); }
        if (slot < r.nQH + r.nKVH) {
            const float y0 = x0 * e.a - x1 * e.b, y1 = x1 * e.a + x0 * e.b;
            x0 = y0; x1 = y1;
        }
        T* dst;
        if (slot < r.nQH) dst = static_cast<T*>(a.out) + size_t(m) * a.ldo + size_t(slot) * r.D;
        else {
            const int pos = r.pos_dev ? min(*r.pos_dev, r.max_seq - 1) : r.pos0;
            const bool is_k = slot < r.nQH + r.nKVH;
            const int kvh = slot - r.nQH - (is_k ? 0 : r.nKVH);
            dst = static_cast<T*>(is_k ? r.kcache : r.vcache) + ((size_t(m) * r.nKVH + kvh) * r.max_seq + pos) * r.D;
        }
        dst[d] = from_float<T>(x0); dst[d + half] = from_float<T>(x1);
    } else if (EPI == EPI_PAIRROT) {
        const SkinnyPairRot& r = a.pair;
        const int grp = tile * (kStcRows / 16) + p / 8, per_head = r.plain + r.rotated, head = grp * 16 / per_head, j = grp * 16 % per_head, i = p % 8;
        if (head >= r.heads) return;
        if (j < r.plain) {
            T* row = static_cast<T*>(a.out) + size_t(m) * a.ldo + size_t(head) * r.plain + j + i;
            row[0] = from_float<T>(x0); row[8] = from_float<T>(x1);
        } else {
            T* row = static_cast<T*>(r.rot_out) + (size_t(m) * r.heads + head) * r.rot_ld + r.rot_col + (j - r.plain) + i;
            row[0] = from_float<T>(x0 * e.a - x1 * e.b); row[8] = from_float<T>(x1 * e.a + x0 * e.b);
        }
    } else {
        #pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int n = tile * kStcRows + p + kStcPairs * h;
            const float v = h ? x1 : x0;
            if (n < a.N) {
                const size_t idx = size_t(m) * a.ldo + n;
                if (EPI == EPI_STORE16)      static_cast<T*>(a.out)[idx] = from_float<T>(v);
                else if (EPI == EPI_STORE32) static_cast<float*>(a.out)[idx] = v;
                else if (EPI == EPI_ADD_FOLD) {
                    const float x = (h ? e.b : e.a) + v;
                    static_cast<float*>(a.out)[idx] = x;
                    static_cast<T*>(a.fold.x16)[size_t(m) * a.N + n] = from_float<T>(x * (h ? e.d : e.c));
                    *sq += x * x;
                }
                else                         static_cast<float*>(a.out)[idx] = (h ? e.b : e.a) + v;
            }
        }
    }
}

// Columns [64 * blk0, 64 * (blk0 + nblk)) of X from the fp32 residual stream into swizzled 16-bit blocks of NB rows
// (PRO_RMSNORM, PRO_POSTADD).  The rows' sums of squares meet over the cluster in `ss` [Mp][CS * warps per row].
template <typename T, int PRO, int NB>
__device__ __forceinline__ void stc_prologue(const SkinnyArgs& a, unsigned char* xs, float* ss, uint64_t* ss_bar, int CS, int rank, bool first_cluster,
                                             int blk0, int nblk, int warp, int lane, int* status, bool& ok) {
    constexpr int CACHE = NB == 16 || PRO == PRO_POSTADD ? 4 : 8;      // quads per lane and row held between the sum and the scaling
    constexpr int ROWS = NB / 8;                             // rows per warp when there is a warp or less per row
    const int K = a.K;
    const int Mp = NB == 16 ? 16 : a.M <= 1 ? 1 : a.M <= 2 ? 2 : a.M <= 4 ? 4 : 8;
    const int wpr = Mp >= 8 ? 1 : 8 / Mp, part = warp % wpr, row0 = warp / wpr;
    const int quads = nblk * (kStcBlock / 4), step = 32 * wpr;
    const T* nw = static_cast<const T*>(a.norm_w);
    const int c0 = blk0 * kStcBlock;
    const int ldx = PRO == PRO_RMSNORM && a.ldx32 ? a.ldx32 : K;
    const bool summed = PRO == PRO_RMSNORM || a.Y32 != nullptr;
    auto live = [&](int q) { return q < quads && c0 + 4 * q < K; };
    auto src = [&](const float* base, int m, int q) { return *reinterpret_cast<const float4*>(base + size_t(m) * ldx + c0 + 4 * q); };
    const float* sq = PRO == PRO_RMSNORM ? a.X32 : a.Y32;    // what the norm is over
    float4 cx[ROWS][CACHE], cy[PRO == PRO_POSTADD ? ROWS : 1][PRO == PRO_POSTADD ? CACHE : 1];
    uint2 cw[CACHE];
    #pragma unroll
    for (int it = 0; it < CACHE; ++it) {
        const int q = part * 32 + lane + it * step;
        cw[it] = make_uint2(0u, 0u);
        if (summed && live(q)) cw[it] = *reinterpret_cast<const uint2*>(nw + c0 + 4 * q);
        #pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const int m = row0 + 8 * r;
            cx[r][it] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (m < a.M && live(q)) cx[r][it] = src(a.X32, m, q);
            if constexpr (PRO == PRO_POSTADD) {
                cy[r][it] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (summed && m < a.M && live(q)) cy[r][it] = src(a.Y32, m, q);
            }
        }
    }
    float inv[ROWS];
    #pragma unroll
    for (int r = 0; r < ROWS; ++r) inv[r] = 0.f;
    if (summed) {
        #pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const int m = row0 + 8 * r;
            float s = 0.f;
            #pragma unroll
            for (int it = 0; it < CACHE; ++it) {
                float4 v;
                if constexpr (PRO == PRO_POSTADD) v = cy[r][it]; else v = cx[r][it];
                s += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
            }
            if (m < a.M)
                for (int q = part * 32 + lane + CACHE * step; live(q); q += step) {
                    const float4 v = src(sq, m, q);
                    s += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
                }
            s = wave::dpp::reduce_sum(s);
            if (lane < CS)
                st_async_f32(cluster_addr(dme::smem_addr(ss + (size_t(m) * CS + rank) * wpr + part), uint32_t(lane)), s,
                             cluster_addr(dme::smem_addr(ss_bar), uint32_t(lane)));
        }
        if (ok && !dme::wait<true>(ss_bar, 0, status)) ok = false;
        __syncwarp();
        #pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const int m = row0 + 8 * r, n = CS * wpr;
            float s = 0.f;
            for (int i = lane; i < n; i += 32) s += ss[size_t(m) * n + i];
            s = wave::dpp::reduce_sum(s);
            inv[r] = rsqrtf(s / float(a.norm_n ? a.norm_n : K) + a.eps);
        }
    }
    auto put = [&](int r, int q, const float4& x, const float4& y, const uint2& wq) {
        const int m = row0 + 8 * r;
        const T* w = reinterpret_cast<const T*>(&wq);
        float4 o = x;
        if (PRO == PRO_RMSNORM) {
            o.x = x.x * inv[r] * to_float(w[0]); o.y = x.y * inv[r] * to_float(w[1]);
            o.z = x.z * inv[r] * to_float(w[2]); o.w = x.w * inv[r] * to_float(w[3]);
        } else if (summed) {
            o.x += y.x * inv[r] * to_float(w[0]); o.y += y.y * inv[r] * to_float(w[1]);
            o.z += y.z * inv[r] * to_float(w[2]); o.w += y.w * inv[r] * to_float(w[3]);
            if (first_cluster && live(q)) *reinterpret_cast<float4*>(a.x_out + size_t(m) * K + c0 + 4 * q) = o;
        }
        const int blk = q / 16, chunk = (q % 16) / 2;
        *reinterpret_cast<uint2*>(xs + blk * (NB * 128) + r * 1024 + row0 * 128 + ((chunk ^ row0) * 16) + (q % 2) * 8) =
            make_uint2(pack2<T>(o.x, o.y), pack2<T>(o.z, o.w));
    };
    #pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        if (row0 + 8 * r >= a.M) continue;                   // zero rows were cleared ahead of the dependency wait
        #pragma unroll
        for (int it = 0; it < CACHE; ++it) {
            const int q = part * 32 + lane + it * step;
            if (q < quads) {
                if constexpr (PRO == PRO_POSTADD) put(r, q, cx[r][it], cy[r][it], cw[it]);
                else put(r, q, cx[r][it], cx[r][it], cw[it]);
            }
        }
        for (int q = part * 32 + lane + CACHE * step; q < quads; q += step) {
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
            uint2 wq = make_uint2(0u, 0u);
            if (live(q)) {
                x = src(a.X32, row0 + 8 * r, q);
                if (PRO == PRO_POSTADD && summed) y = src(a.Y32, row0 + 8 * r, q);
                if (summed) wq = *reinterpret_cast<const uint2*>(nw + c0 + 4 * q);
            }
            put(r, q, x, y, wq);
        }
    }
}

template <typename T, int PRO, int EPI, int NB>
__global__ void __launch_bounds__(kStcThreads, 2)
skinny_tc_kernel(const SkinnyArgs a, const SkinnyTcShape sh, const __grid_constant__ CUtensorMap mapW, const __grid_constant__ CUtensorMap mapX,
                 int* status, int* sticky) {
    griddep_launch_dependents();
    extern __shared__ __align__(1024) unsigned char stc_raw[];
    unsigned char* const stc_smem = stc_raw + (-dme::smem_addr(stc_raw) & 1023u);      // swizzle atoms start on 1 KB, wherever the linker put the array
    __shared__ uint64_t full[kStcMaxStages], empty[kStcMaxStages], prod_full[kStcSlots], prod_empty[kStcSlots], inbox_full[2], x_full, ss_full, drained;
    __shared__ __align__(16) float ss[16 * kStcMaxCluster];
    static_assert(kStcWorkers == kSkinnyThreads, "fold_inverse");
    __shared__ float inv_rms[PRO == PRO_SCALED ? 16 : 1];
    __shared__ uint32_t s_tmem;
    constexpr int ROW = stc_inbox_row(NB);
    constexpr int AHEAD = kStcPairs * NB / kStcWorkers;          // (pair, row) items of a thread when one CTA owns the whole tile
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int CS = sh.cluster, rank = int(blockIdx.x) % CS, cluster = int(blockIdx.x) / CS, nclusters = int(gridDim.x) / CS;
    const int blk0 = rank * sh.kblocks / CS, nblk = (rank + 1) * sh.kblocks / CS - blk0;
    const int per = (kStcPairs + CS - 1) / CS;                   // pairs per owner
    unsigned char* xs = stc_smem;
    unsigned char* stages = stc_smem + sh.x_bytes;
    float* inbox = reinterpret_cast<float*>(stages + size_t(sh.nstages) * kStcStageBytes);   // [2][CS][2 * per][ROW] (one buffer if there is one tile)
    const int inbox_floats = sh.inbox_bytes / 4;
    float* squares = inbox + (sh.ntiles > nclusters ? 2 : 1) * inbox_floats;                 // EPI_ADD_FOLD: as many buffers of [NB][per]

    if (threadIdx.x == 0) {
        for (int s = 0; s < sh.nstages; ++s) { dme::mbar_init(&full[s], 1); dme::mbar_init(&empty[s], 1); }
        for (int b = 0; b < kStcSlots; ++b) { dme::mbar_init(&prod_full[b], 1); dme::mbar_init(&prod_empty[b], kStcWorkers / 32); }
        for (int b = 0; b < 2; ++b) dme::mbar_init(&inbox_full[b], 1);
        dme::mbar_init(&x_full, pro_rows16(PRO) ? 1 : kStcWorkers);
        dme::mbar_init(&ss_full, 1);
        dme::mbar_init(&drained, 1);
        dme::mbar_init_fence();
    }
    if (warp == kStcWorkers / 32 + 1) { tc::tmem_alloc(&s_tmem, kStcTmemCols); tc::tmem_relinquish(); }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = s_tmem;
    // the cluster's barriers exist once this has completed; whoever writes to a peer waits for it first
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    bool ok = true;

    if (warp == kStcWorkers / 32) {
        // ---- producer ------------------------------------------------------------------------------------------
        if (lane == 0) {
            dme::prefetch_tensor_map(&mapW);
            const uint64_t pol = dme::policy_evict_first();
            int stage = 0, uses = 0; uint32_t phase = 0;
            bool x_asked = !pro_rows16(PRO);
            auto ask_x = [&] {                                    // the slice of X, once the kernels before have finished
                griddep_wait();                                   // (makes the kernels' writes visible to the copies too)
                dme::mbar_arrive_expect_tx(&x_full, uint32_t(nblk) * (NB * 128));
                for (int b = 0; b < nblk; ++b) dme::copy_tile_2d(xs + b * (NB * 128), &mapX, (blk0 + b) * kStcBlock, 0, &x_full);
                x_asked = true;
            };
            for (int tile = cluster; tile < sh.ntiles && ok; tile += nclusters) {
                for (int b = 0; b < nblk; ++b) {
                    if (uses >= sh.nstages) {
                        if (!x_asked) ask_x();                    // the ring is full: nothing left to do ahead of the wait
                        if (!dme::wait(&empty[stage], phase ^ 1u, status)) { ok = false; break; }
                    }
                    const int x = (blk0 + b) * kStcBlock;
                    unsigned char* dst = stages + size_t(stage) * kStcStageBytes;
                    dme::mbar_arrive_expect_tx(&full[stage], kStcStageBytes);
                    if (epi_gated(EPI)) {
                        dme::copy_tile_2d_stream(dst, &mapW, x, tile * kStcPairs, &full[stage], pol);
                        dme::copy_tile_2d_stream(dst + kStcStageBytes / 2, &mapW, x, a.N + tile * kStcPairs, &full[stage], pol);
                    } else {
                        dme::copy_tile_2d_stream(dst, &mapW, x, tile * kStcRows, &full[stage], pol);
                    }
                    ++uses; if (++stage == sh.nstages) { stage = 0; phase ^= 1u; }
                }
            }
            if (!x_asked) ask_x();
            if (!ok) {
                // the copies in flight land before this CTA's shared memory is given up
                for (int i = 0; i < min(uses, sh.nstages); ++i) {
                    const int u = uses - 1 - i;
                    dme::wait(&full[u % sh.nstages], uint32_t(u / sh.nstages) & 1u);
                }
                if (pro_rows16(PRO)) dme::wait(&x_full, 0);
                atomicExch(sticky, 1);
            }
        }
        __syncwarp();
    } else if (warp == kStcWorkers / 32 + 1) {
        // ---- MMA issuer: all lanes walk the loop, one issues (tc::elect_one) --------------------------------------
        constexpr uint32_t idesc = tc::instr_desc_f16(kStcRows, NB, StcFmt<T>::id, 0, 0);
        int stage = 0, use = 0; uint32_t phase = 0;
        auto wait = [&](uint64_t* bar, uint32_t parity) { ok = __all_sync(0xffffffffu, dme::wait(bar, parity, status)) != 0; return ok; };
        const uint64_t a0 = tc::smem_desc_sw128(dme::smem_addr(stages), 16, 1024), b0 = tc::smem_desc_sw128(dme::smem_addr(xs), 16, 1024);
        wait(&x_full, 0);
        // the blocks take the slots in turn; what was in a slot before must have been read
        auto slot_parity = [](int u) { return uint32_t(u / kStcSlots - 1) & 1u; };
        bool bytes = false, room = true;                          // seen to be there, asked ahead of the MMAs before:
        for (int tile = cluster; tile < sh.ntiles && ok; tile += nclusters) {             // a wait takes 130 cycles even when there is nothing to wait for
            for (int k = 0; k < nblk; ++k) {
                const int slot = use % kStcSlots;
                if (!bytes && !wait(&full[stage], phase)) break;
                if (!room && !wait(&prod_empty[slot], slot_parity(use))) break;
                tc::fence_after_sync();
                const uint64_t ad = a0 + uint64_t(stage * (kStcStageBytes / 16)), bd = b0 + uint64_t(k * (NB * 128 / 16));
                uint64_t* const freed = &empty[stage];
                ++use;
                if (++stage == sh.nstages) { stage = 0; phase ^= 1u; }
                const bool next_bytes = dme::mbar_test_wait(&full[stage], phase);
                const bool next_room = use < kStcSlots || dme::mbar_test_wait(&prod_empty[use % kStcSlots], slot_parity(use));
                if (tc::elect_one()) {
                    #pragma unroll
                    for (int s = 0; s < 4; ++s)
                        tc::mma_ss(tmem + slot * kStcSlotCols + s * kStcAccs / 4 * 16, ad + uint64_t(s * 2), bd + uint64_t(s * 2), idesc, s * kStcAccs % 4 != 0);
                    tc::commit(freed);
                    tc::commit(&prod_full[slot]);
                }
                bytes = __all_sync(0xffffffffu, next_bytes) != 0;
                room = __all_sync(0xffffffffu, next_room) != 0;
            }
        }
        if (!ok) {                                                // the products in flight end before tensor memory is freed
            if (tc::elect_one()) { tc::commit(&drained); atomicExch(sticky, 1); }
            dme::wait(&drained, 0);
        }
        __syncwarp();
    } else {
        // ---- workers: X, then the exchange and the epilogue ------------------------------------------------------
        const int tid = threadIdx.x;
        const int mine = max(0, min(per, kStcPairs - rank * per)); // pairs this CTA owns
        if (!pro_rows16(PRO)) {
            if (a.M < NB) {                                       // rows past M
                for (int i = tid; i < nblk * (NB * 8); i += kStcWorkers)
                    if ((i / 8) % NB >= a.M) *reinterpret_cast<uint4*>(xs + size_t(i) * 16) = make_uint4(0u, 0u, 0u, 0u);
            }
            if (tid == 0 && (PRO == PRO_RMSNORM || a.Y32)) dme::mbar_arrive_expect_tx(&ss_full, uint32_t(NB * CS * 4));
            __syncwarp();
        }
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        griddep_wait();
        if constexpr (PRO == PRO_SCALED) {
            float4 sums[NB / 8][4];
            fold_load(a, warp, lane, sums);
            fold_inverse(a, warp, lane, sums, inv_rms);
            stc_worker_barrier();
        } else if constexpr (PRO != PRO_PLAIN) {
            stc_prologue<T, PRO, NB>(a, xs, ss, &ss_full, CS, rank, cluster == 0, blk0, nblk, warp, lane, status, ok);
            dme::fence_proxy_async_smem();
            dme::mbar_arrive(&x_full);
        }
        constexpr int HB = NB / 2;
        const int quarter = warp % 4, h = warp / 4;               // TMEM lanes of the warp; half of the NB columns
        const int2 pr = stc_pair<EPI>(a, 32 * quarter + lane);
        const int owner = pr.x / per, row = (pr.x % per) * 2 + pr.y;
        int it = 0, use = 0;
        for (int tile = cluster; tile < sh.ntiles; tile += nclusters, ++it) {
            const int b = it & 1;
            float* box = inbox + b * inbox_floats;
            if (tid == 0) dme::mbar_arrive_expect_tx(&inbox_full[b], uint32_t(mine) * 2 * NB * 4 * CS);
            StcAhead ahead[AHEAD];
            #pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
                const int idx = tid + u * kStcWorkers;
                if (idx < mine * NB) ahead[u] = stc_fetch<T, EPI>(a, tile, rank * per + idx % mine, idx / mine);
            }
            // the blocks' products, in two sums that take turns
            float sum[HB], other[HB];
            #pragma unroll
            for (int j = 0; j < HB; ++j) sum[j] = other[j] = 0.f;
            for (int k = 0; k < nblk; ++k, ++use) {
                const int slot = use % kStcSlots;
                if (ok && !dme::wait(&prod_full[slot], uint32_t(use / kStcSlots) & 1u, status)) ok = false;
                __syncwarp();
                tc::fence_after_sync();
                uint32_t v[kStcAccs][HB];
                #pragma unroll
                for (int s = 0; s < kStcAccs; ++s) tc::ld_32x32b<HB>(tc::tmem_addr(tmem, 32 * quarter, slot * kStcSlotCols + s * 16 + h * HB), v[s]);
                tc::wait_ld();
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) dme::mbar_arrive(&prod_empty[slot]);
                #pragma unroll
                for (int j = 0; j < HB; ++j) {
                    const float next = sum[j] + (__uint_as_float(v[0][j]) + __uint_as_float(v[1][j]));
                    sum[j] = other[j]; other[j] = next;
                }
            }
            uint32_t v[HB];
            #pragma unroll
            for (int j = 0; j < HB; ++j) v[j] = __float_as_uint(sum[j] + other[j]);
            {
                const uint32_t dst = cluster_addr(dme::smem_addr(box + (size_t(rank) * 2 * per + row) * ROW + h * HB), uint32_t(owner));
                const uint32_t bar = cluster_addr(dme::smem_addr(&inbox_full[b]), uint32_t(owner));
                #pragma unroll
                for (int j = 0; j < NB / 8; ++j) st_async_v4(dst + 16 * j, v + 4 * j, bar);
            }
            if (ok && !dme::wait<true>(&inbox_full[b], uint32_t((it >> 1) & 1), status)) ok = false;
            #pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
                const int idx = tid + u * kStcWorkers;
                if (idx < mine * NB) {
                    const int p = idx % mine, m = idx / mine;
                    float x0 = 0.f, x1 = 0.f;
                    for (int s = 0; s < CS; ++s) {
                        const float* part = box + (size_t(s) * 2 * per + 2 * p) * ROW + m;
                        x0 += part[0]; x1 += part[ROW];
                    }
                    if (PRO == PRO_SCALED) { x0 *= inv_rms[m]; x1 *= inv_rms[m]; }
                    stc_epilogue<T, EPI>(a, tile, rank * per + p, m, x0, x1, ahead[u], squares + b * NB * per + idx);
                }
            }
            stc_worker_barrier();
            // (the buffer is written again two tiles on, behind the next tile's barrier)
            if (EPI == EPI_ADD_FOLD && tid < a.M) {
                const float* sq = squares + b * NB * per + tid * mine;
                float s = 0.f;
                for (int p = 0; p < mine; ++p) s += sq[p];
                a.fold.ss_out[size_t(tid) * a.fold.ss_ld + tile * CS + rank] = s;
            }
        }
        if (!ok && lane == 0) atomicExch(sticky, 1);
        __syncwarp();
    }
    // nobody leaves while a peer may still write here
    if (warp >= kStcWorkers / 32) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    tc::fence_after_sync();
    if (warp == kStcWorkers / 32 + 1) tc::tmem_dealloc(tmem, kStcTmemCols);
}

// Whether the shape is in the domain of this kernel and the other two: K a multiple of 16 (32-byte steps along the rows of W
// and X), ldx of 8, W 16-byte aligned (bulk copies and tensor maps).
template <int PRO, int EPI>
bool skinny_domain(const SkinnyArgs& a) {
    if (a.M < 1 || a.M > kSkinnyMaxM || a.K < 16 || a.K % 16 != 0 || a.N < 1 || !aligned(a.W, 16)) return false;
    if (pro_rows16(PRO) && (a.ldx % 8 != 0 || !aligned(a.X16, 16))) return false;
    if (PRO == PRO_SCALED && (a.fold.parts < 1 || !aligned(a.fold.ss, 16) || a.fold.ss_ld % 4 != 0)) return false;
    if (PRO == PRO_RMSNORM && (!aligned(a.X32, 16) || !aligned(a.norm_w, 8) || a.ldx32 % 4 != 0)) return false;
    if (PRO == PRO_POSTADD && (!aligned(a.X32, 16) || !aligned(a.Y32, 16) || !aligned(a.x_out, 16) || !aligned(a.norm_w, 8))) return false;
    if (EPI == EPI_PAIRROT && (a.pair.plain % 16 != 0 || a.pair.rotated % 16 != 0 || a.N != a.pair.heads * (a.pair.plain + a.pair.rotated))) return false;
    return EPI != EPI_ROPE || (a.rope.D % 16 == 0 && a.N == (a.rope.nQH + 2 * a.rope.nKVH) * a.rope.D);
}

// Clusters of `cluster` CTAs that run at the same time on the current device, one CTA per SM; 0 if it cannot be learnt now.
int stc_resident_clusters(int cluster);

// Clusters that run at a time if `cs` CTAs may share `blocks` blocks of K: 0 where a slice of X does not fit beside the ring,
// where the knob says another number (no more than there are blocks) or where the device runs no such cluster.
constexpr int kStcMaxXBytes = 136 * 1024;
inline int stc_clusters(int cs, int blocks, int rows) {
    const int forced = tuning(KNOB_SKINNY_CLUSTER, 0);
    if (cs > blocks || (forced > 0 && cs != (forced < blocks ? forced : blocks))) return 0;
    return (blocks + cs - 1) / cs * rows * 128 <= kStcMaxXBytes ? stc_resident_clusters(cs) : 0;
}
// Whether some split of K serves M rows: what decides between the decode kernels and the GEMM ahead of any launch.
inline bool skinny_tc_fits(int M, int K) {
    for (int cs = 1; cs <= kStcMaxCluster && M <= kSkinnyMaxM; ++cs)
        if (stc_clusters(cs, (K + kStcBlock - 1) / kStcBlock, M <= 8 ? 8 : 16) > 0) return true;
    return false;
}
// Whether M rows of K columns against a W of `bytes` take the kernel of this file rather than those of skinny_gemm.cuh: where X
// does not fit those, or leaves their ring no second stage of weights (more than 96 KB of X: 16 rows of 3073 columns, 8 of 6145, 4 of
// 12289).  Projections launched one after the other as a decode step does it, cold W, the other kernels against this one:
//   16 rows, O of 4096 columns 18.4 -> 11.3 us; gate/up of 4096 x 4096 40.8 -> 20.5; down of 2048 x 5632 18.3 -> 10.4; head of
//   2048 x 3200 19.4 -> 9.2; 8 rows, 4096 x 8192 29.5 -> 17.9; and on this side of the line, where they are the faster ones,
//   16 rows of 2048 columns: gate/up of 4096 11.9 against 15.6, head of 32000 26.2 against 29.9; 8 rows, 2048 x 5632 7.3 against 9.2.
// Of 500 shapes two are slower beyond the line (9 rows, 512 and 1024 x 4096: 5.4 against 5.7 and 5.9 against 6.1 us).
// A call without an abort word of its own clears one by a memset first, which ends the overlap with the launch before, 4 us
// that the register kernel does not need: then only from 20 MB of W on with 9 to 16 rows (2048 x 5632: 18.4 -> 14.5 us, but
// 1024 x 5632 9.3 against 12.4) and from 64 MB on with fewer (8192 x 6400: 29.8 -> 28.0, but 4096 x 6400 16.6 against 18.8).
inline bool skinny_split(int M, int K, size_t bytes, bool own_abort_word) {
    const int Mp = M <= 1 ? 1 : M <= 2 ? 2 : M <= 4 ? 4 : M <= 8 ? 8 : 16;
    if (!skinny_rows_fit(M, K)) return true;
    return size_t(Mp) * K * 2 > 96 * 1024 && (own_abort_word || bytes > size_t(M > 8 ? 20 : 64) << 20);
}

// Whether M rows of K columns run on a kernel that has the folded forms (this file's or the streaming one: the register kernel has
// none), for a caller with an abort word of its own.  Holds for fewer columns too where it holds for K.
inline bool skinny_folds(int M, int K) {
    const int kind = tuning(KNOB_RUNTIME_SKINNY, 2);
    if (M > kSkinnyMaxM || kind < 2) return false;
    if ((kind == 3 || skinny_split(M, K, 0, true)) && skinny_tc_fits(M, K)) return true;
    return kind == 2 && skinny_rows_fit(M, K) && skinny_ring(M, K).nstages >= 2;
}

// B200P_E_RANGE: the shape is outside the kernel's domain (nothing was launched).
template <typename T, int PRO, int EPI, int NB>
int launch_skinny_tc(const SkinnyArgs& a, cudaStream_t st, int* parts = nullptr) {
    const int tiles = epi_gated(EPI) ? (a.N + kStcPairs - 1) / kStcPairs : (a.N + kStcRows - 1) / kStcRows;
    if (EPI == EPI_ROPE && a.rope.D != 64 && a.rope.D != 128) return B200P_E_RANGE;
    SkinnyTcShape sh{};
    sh.kblocks = (a.K + kStcBlock - 1) / kStcBlock;
    sh.ntiles = tiles;
    // The split of K that moves the fewest bytes through the busiest CTA: rounds of tiles times blocks per slice, plus
    // what a round costs apart from the stream (in blocks of 16 KB; an SM streams one in 0.36 us).  A norm prologue holds
    // the residual of 16 blocks (8 with more than 8 rows) in registers; what it has to read again counts half a block each.
    // Against the best of all sizes, forced, for shapes that take this kernel: 4 to 16 rows, O, gate/up, down and head of width 4096,
    // down of 2048: within 3 %, gate/up with 4 and 8 rows 5 %; Q/K/V of width 4096 with 16 rows 22.9 us against 21.0 with 8.
    int best = 0, clusters = 0;
    long long best_cost = 0;
    for (int cs = 1; cs <= kStcMaxCluster; ++cs) {
        const int res = stc_clusters(cs, sh.kblocks, NB);
        if (res < 1) continue;
        const int slice = (sh.kblocks + cs - 1) / cs, rounds = (tiles + res - 1) / res;
        const long long cost = (long long)(rounds) * (slice + 1) + (slice > 16 && !pro_rows16(PRO) ? (slice - 16) / 2 : 0);
        if (!best || cost < best_cost) { best = cs; best_cost = cost; clusters = tiles < res ? tiles : res; }
    }
    if (!best) return B200P_E_RANGE;
    sh.cluster = best;
    const int slice = (sh.kblocks + best - 1) / best, per = (kStcPairs + best - 1) / best;
    sh.x_bytes = slice * NB * 128;
    sh.inbox_bytes = best * 2 * per * stc_inbox_row(NB) * 4;
    const int uses = slice * ((tiles + clusters - 1) / clusters);
    // less than half an SM's shared memory if that leaves four stages
    const int boxes = tiles > clusters ? 2 : 1, squares = EPI == EPI_ADD_FOLD ? NB * per * 4 : 0, fixed = sh.x_bytes + boxes * (sh.inbox_bytes + squares);
    int nst = (110 * 1024 - fixed) / kStcStageBytes;
    if (nst < 4 && nst < uses) nst = (223 * 1024 - fixed) / kStcStageBytes;
    nst = nst > kStcMaxStages ? kStcMaxStages : nst;
    sh.nstages = nst > uses ? uses : nst;
    if (sh.nstages < 1) return B200P_E_RANGE;
    int* sticky = device_status_ptr();
    if (!sticky) return B200P_E_RANGE;
    const CUtensorMapDataType dt = StcFmt<T>::id ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    CUtensorMap mw, mx;
    const uint64_t rows = uint64_t(a.N) * (epi_gated(EPI) ? 2 : 1);
    const uint64_t wd[2] = {uint64_t(a.K), rows}, ws[1] = {uint64_t(a.K) * 2};
    const uint32_t wbox[2] = {uint32_t(kStcBlock), uint32_t(epi_gated(EPI) ? kStcPairs : kStcRows)};
    if (cudaError_t e = make_tensor_map(&mw, dt, 2, a.W, wd, ws, wbox, Swizzle::B128)) return int(e);
    mx = mw;
    if (pro_rows16(PRO)) {
        const uint64_t xd[2] = {uint64_t(a.K), uint64_t(a.M)}, xst[1] = {uint64_t(a.ldx) * 2};
        const uint32_t xbox[2] = {uint32_t(kStcBlock), uint32_t(NB)};
        if (cudaError_t e = make_tensor_map(&mx, dt, 2, a.X16, xd, xst, xbox, Swizzle::B128)) return int(e);
    }
    int* status = a.abort_word;
    if (!status) {
        LaunchSlot slot{};
        if (int se = take_launch_slot(st, &slot)) return se;
        status = slot.abort;
    }
    size_t dyn = 1024 + size_t(sh.x_bytes) + size_t(sh.nstages) * kStcStageBytes + size_t(boxes) * (sh.inbox_bytes + squares);
    if (dyn < size_t(kStcMinDynamic)) dyn = size_t(kStcMinDynamic);
    auto kern = skinny_tc_kernel<T, PRO, EPI, NB>;
    if (int e = allow_dynamic_smem(reinterpret_cast<const void*>(kern), dyn)) return e;
    if (parts) *parts = tiles * best;
    return launch_dependent_clusters(kern, best, dim3(unsigned(clusters * best)), kStcThreads, dyn, st, a, sh, mw, mx, status, sticky);
}

// Launch: returns B200P_E_RANGE when the shape is outside the kernels' domain (the caller then takes the GEMM).
// *parts: the partial sums of EPI_ADD_FOLD, at most fold_parts_most (one per eight columns, or CTA of a cluster and tile).
inline int fold_parts_most(int N) { return (N + kStcRows - 1) / kStcRows * (kStcRows / 8); }
static_assert(kStcMaxCluster <= kStcRows / 8);
template <typename T, int PRO, int EPI>
int launch_skinny(const SkinnyArgs& a, cudaStream_t st, int* parts = nullptr) {
    if (!skinny_domain<PRO, EPI>(a)) return B200P_E_RANGE;
    const int kind = tuning(KNOB_RUNTIME_SKINNY, 2);
    if (kind == 3 || (kind == 2 && skinny_split(a.M, a.K, size_t(a.N) * a.K * (epi_gated(EPI) ? 4 : 2), a.abort_word != nullptr))) {
        const int e = a.M <= 8 ? launch_skinny_tc<T, PRO, EPI, 8>(a, st, parts) : launch_skinny_tc<T, PRO, EPI, 16>(a, st, parts);
        if (kind == 3 || e != B200P_E_RANGE) return e;
    }
    // up to 8 rows of X: one B fragment per A fragment; 9 .. 16 rows: two
    return a.M <= 8 ? launch_skinny_mh<T, PRO, EPI, 1>(a, st, parts) : launch_skinny_mh<T, PRO, EPI, 2>(a, st, parts);
}

} // namespace b200p
