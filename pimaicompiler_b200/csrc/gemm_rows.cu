// Dense contraction with fused epilogues on the 5th-generation tensor cores, activation rows as the M operand:
//
//     D[j, n] = sum_k X[j, k] W[n, k]   (both K-major; optionally a second pair X2, W2 whose products join the same sums)
//
// Activation rows are TMEM lanes and weight rows TMEM columns, so an epilogue thread owns one activation row and walks its
// outputs in registers: bias / ReLU, the arg max over a vocabulary or the gates of an LSTM cell need no exchange between
// threads.
//
// What bounds it: operands reach an SM at about 64 bytes per cycle (from L2), and a 128 x BN tile of one CTA needs
// (128 + BN) * 128 bytes per K block of 64, which its MMAs use up in 2 * BN cycles: 128 x 128 waits for operands half the
// time, 128 x 256 a third.  So two CTAs on neighbouring SMs share a tile (cta_group::2): each loads its own 128 activation
// rows and half of the BN weight rows, the pair multiplies 256 x BN, and at BN = 256 an SM's 32 KB per K block last the
// 512 cycles they take to load.  Products with few tiles take a smaller BN, and single CTAs, which spreads them over more SMs (pick).
//
// Persistent CTA pairs, warp-specialised: warps 0 and 1 TMA producers (in both CTAs; all bytes of a stage are counted by
// the leader's barrier), warp 2 TMEM owner and, in the leader, MMA issuer for the pair, warps 3..10 the epilogue of the
// CTA's own rows (two warps per TMEM lane quarter, each with every second chunk of columns), two accumulator stages.  fp16 and
// fp32 outputs leave through shared memory and TMA stores, each warp on its own 32 rows (a thread's own stores would
// touch one 32-byte sector in each of 32 rows).  Every mbarrier wait is bounded; when one runs out the kernel records an
// error in the status word, lets outstanding bulk copies land (bounded), frees its TMEM and returns.
#include "gemm_rows.cuh"

#include <mutex>

#include "common.cuh"
#include "tc_common.cuh"

namespace pimb200 {
namespace tc {

namespace {

constexpr int BM = 128;            // activation rows per CTA (UMMA M)
constexpr int BK = 64;             // halves per stage along K = one 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int EPI_WARPS = 8;
constexpr int FIRST_EPI = 3;       // warps before the epilogue's
constexpr int THREADS = (FIRST_EPI + EPI_WARPS) * 32;
constexpr int CHUNK_BYTES = 32 * 128;              // one chunk of outputs: a warp's 32 rows x 128 bytes
constexpr int STAGING_BYTES = EPI_WARPS * 2 * CHUNK_BYTES;
constexpr int A_BYTES = BM * BK * 2;

__host__ __device__ constexpr int b_bytes(int bn, int cg) { return bn / cg * BK * 2; }
// K blocks per pipeline stage.  A wait on a barrier costs 200 cycles even when it is met, so where a K block's MMAs take
// less than twice that, a stage holds two.
__host__ __device__ constexpr int kblocks_for(int bn, int cg) { return bn == 256 || (bn == 128 && cg == 1) ? 1 : 2; }
// As deep as shared memory allows: a stage comes round about 2700 cycles after it was freed (measured with three stages of
// 24 KB), so 64 bytes per cycle need some 170 KB in flight.
__host__ __device__ constexpr int stages_for(int bn, int cg) {
    return cg == 2 ? (bn == 256 ? 5 : (bn == 128 ? 3 : 4)) : (bn == 256 ? 3 : (bn == 128 ? 5 : 3));
}
constexpr size_t smem_for(int bn, int cg) {
    return (size_t)stages_for(bn, cg) * kblocks_for(bn, cg) * (A_BYTES + b_bytes(bn, cg)) + STAGING_BYTES + 1024 /*align*/ + 256 /*barriers*/;
}
static_assert(smem_for(256, 2) <= 232448 && smem_for(256, 1) <= 232448 && smem_for(128, 2) <= 232448 &&
              smem_for(128, 1) <= 232448 && smem_for(64, 2) <= 232448 && smem_for(64, 1) <= 232448, "fits one SM");

struct Maps {
    CUtensorMap x, w, x2, w2, y, y_tail;   // y: boxes of 32 rows; y_tail: of the jrows % 32 rows behind the last whole 32
};

struct Args {
    const __half* bias;       // [N] or NULL (outputs and arg max)
    int N, J, act;
    int jrows;                // activation rows per CTA: 128, or J if it is less, or the whole timesteps that fit in 128 rows
    int bn;                   // weight rows per tile: a multiple of 32 (64 for the cell), at most the template's BN
    int kb1, kb2;             // K blocks of 64 of the first and the second pair
    int j_tiles, n_tiles;     // tiles along the activation rows (of one CTA or a pair) and along the weight rows
    void* Y;
    long ldy;
    int direct;               // 1: the outputs are stored by the warps, row by row; 2: and rows start at multiples of 4 bytes
    int fixed;                // 1: no work ahead on the stream writes the weights (they may be read before that work has ended)
    int x_batch;              // > 0: rows are numbered time-major over batch-first sequences (map x is 3-D: K, b, t)
    int* status;
    int gen;
    // arg max: best value and its index of each (column half of a tile, row)
    float* best_v;            // [2 * n_tiles][J]
    int* best_i;
    // LSTM cell
    const float* cell_bias;   // packed [4H]
    const __half* c0;         // [J, H] or NULL
    __half* y;                // row j at y + j * y_ld
    long y_ld;
    __half* hn;               // [J, H] or NULL
    __half* cn;
    const __half* res;        // optional residual rows
    long res_ld;
    int H;
};

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map), "r"(src), "r"(c0),
                 "r"(c1)
                 : "memory");
}
__device__ __forceinline__ void load_half16(const __half* p, float* f) {     // 16 halves, 16-byte aligned
    const uint4* q = reinterpret_cast<const uint4*>(p);
    widen8(q[0], f);
    widen8(q[1], f + 8);
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ void store_half16(__half* p, const uint32_t* w) {
    uint4* q = reinterpret_cast<uint4*>(p);
    q[0] = make_uint4(w[0], w[1], w[2], w[3]);
    q[1] = make_uint4(w[4], w[5], w[6], w[7]);
}

// Rows of a warp's staged chunk (128 bytes each, 16-byte pieces swapped by row) to rows of Y that start at `at`, `ldy` elements apart.
// pairs: every row starts at a multiple of 4 bytes.  Halves eight rows at a time, each lane its own out of shared memory (pairs
// exchanged between lanes, row by row: 33 rows of 2001 x 512 8.1 us, now 6.7).  Not inlined: the kernel's loop has no registers for it
template <bool F32>
__device__ __noinline__ void store_rows(const unsigned char* buf, void* Y, size_t at, long ldy, int rows, int cols, bool pairs) {
    const int lane = threadIdx.x & 31;
    auto piece = [&](int rr, int p) { return buf + rr * 128 + ((p ^ (rr & 7)) << 4); };
    if constexpr (F32) {
#pragma unroll 4
        for (int rr = 0; rr < rows; ++rr, at += ldy) {
            const uint32_t w = *reinterpret_cast<const uint32_t*>(piece(rr, lane >> 2) + (lane & 3) * 4);
            if (lane < cols) static_cast<float*>(Y)[at + lane] = __uint_as_float(w);
        }
        return;
    }
    constexpr int AT_ONCE = 8;             // (the chunk has 32 rows: those behind the last one are read, not stored)
    uint16_t* y = static_cast<uint16_t*>(Y) + at;
    if (pairs) {
        for (int r0 = 0; r0 < rows; r0 += AT_ONCE) {
            uint32_t w[AT_ONCE];
#pragma unroll
            for (int i = 0; i < AT_ONCE; ++i) w[i] = *reinterpret_cast<const uint32_t*>(piece(r0 + i, lane >> 2) + (lane & 3) * 4);
#pragma unroll
            for (int i = 0; i < AT_ONCE; ++i, y += ldy) {
                if (r0 + i >= rows) return;
                if (2 * lane + 1 < cols) *reinterpret_cast<uint32_t*>(y + 2 * lane) = w[i];
                else if (2 * lane < cols) y[2 * lane] = (uint16_t)w[i];
            }
        }
        return;
    }
    for (int r0 = 0; r0 < rows; r0 += AT_ONCE) {
        uint16_t lo[AT_ONCE], hi[AT_ONCE];                 // 2-byte stores of neighbours: lane l takes elements l and 32 + l
#pragma unroll
        for (int i = 0; i < AT_ONCE; ++i) {
            lo[i] = *reinterpret_cast<const uint16_t*>(piece(r0 + i, lane >> 3) + (lane & 7) * 2);
            hi[i] = *reinterpret_cast<const uint16_t*>(piece(r0 + i, 4 + (lane >> 3)) + (lane & 7) * 2);
        }
#pragma unroll
        for (int i = 0; i < AT_ONCE; ++i, y += ldy) {
            if (r0 + i >= rows) return;
            if (lane < cols) y[lane] = lo[i];
            if (32 + lane < cols) y[32 + lane] = hi[i];
        }
    }
}

}  // namespace

template <int BN, int EPI, int CG>
__global__ void __launch_bounds__(THREADS, 1) gemm_rows_kernel(const __grid_constant__ Maps maps, const __grid_constant__ Args a) {
    constexpr int STAGES = stages_for(BN, CG), KS = kblocks_for(BN, CG), B_BYTES = b_bytes(BN, CG);
    constexpr int BLOCK_BYTES = A_BYTES + B_BYTES, STAGE_BYTES = KS * BLOCK_BYTES;
    constexpr int TMEM_COLS = 2 * BN;              // 128, 256 or 512: a power of two
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* staging = smem + (size_t)STAGES * STAGE_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(staging + STAGING_BYTES);
    // bars[0..S) full, [S..2S) empty, [2S..2S+2) accumulator full, [2S+2..2S+4) accumulator empty; then the TMEM base
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + STAGES);
    const uint32_t accf0 = smem_u32(bars + 2 * STAGES), acce0 = smem_u32(bars + 2 * STAGES + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kblocks = a.kb1 + a.kb2;
    const int tiles = a.j_tiles * a.n_tiles;
    const int rank = CG == 2 ? (int)(blockIdx.x & 1) : 0;          // 0 = the leader of the pair
    const int first = blockIdx.x / CG, stride = gridDim.x / CG;    // tiles of this CTA or pair
    const volatile int* abort_flag = a.status + 1;

    if (threadIdx.x == 32) {
        const CUtensorMap* used[] = {&maps.x, &maps.w, &maps.y};
#pragma unroll
        for (int i = 0; i < 3; ++i) asm volatile("prefetch.tensormap [%0];" ::"l"(used[i]) : "memory");
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(accf0 + 8 * s, 1);
            mbar_init(acce0 + 8 * s, CG * EPI_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        if (CG == 1) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                         "r"((uint32_t)TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                         "r"((uint32_t)TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    pair_sync<CG>();                               // the barriers of both CTAs exist before either is signalled
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    bool failed = false;
    pdl_launch_dependents();
    if (warp != 1 || !a.fixed) pdl_wait();

    if (warp < 2) {
        // ---------------- TMA producers: warp 0 the activation rows, warp 1 the weight rows, each one stream of K blocks
        //                  over all tiles of this CTA ----------------
        const uint32_t el = elect_one();
        const uint32_t bytes = (uint32_t)CG * (uint32_t)a.jrows * BK * 2 + (uint32_t)a.bn * BK * 2;   // a K block of both CTAs
        const uint32_t smem0 = smem_u32(smem) + (warp == 0 ? 0 : A_BYTES), lead0 = CG == 1 ? full0 : mapa(full0, 0);
        const bool counts = warp == 0 && rank == 0;            // tells the stage's barrier how many bytes will come
        uint32_t s = 0, par = 1, issued = 0;                   // stage, parity of its "empty" phase, stages issued
        for (int tile = first; tile < tiles && !failed; tile += stride) {
            const int n0 = (tile % a.n_tiles) * a.bn + rank * (a.bn / CG), j0 = ((tile / a.n_tiles) * CG + rank) * a.jrows;
            const int t0 = a.x_batch > 0 ? j0 / a.x_batch : 0;
            for (int k0 = 0; k0 < kblocks; k0 += KS) {
                if (!mbar_wait(empty0 + 8 * s, par, abort_flag, a.gen)) { failed = true; break; }
                const uint32_t bar = lead0 + 8 * s;
                if (counts) expect_tx_if(el, full0 + 8 * s, KS == 1 || k0 + 1 < kblocks ? KS * bytes : bytes);
#pragma unroll
                for (int i = 0; i < KS; ++i) {
                    const int kb = k0 + i, k2 = kb - a.kb1;
                    if (i > 0 && kb >= kblocks) break;
                    const uint32_t dst = smem0 + s * STAGE_BYTES + i * BLOCK_BYTES;
                    if (warp == 1) load_2d<CG>(el, dst, k2 < 0 ? &maps.w : &maps.w2, bar, (k2 < 0 ? kb : k2) * BK, n0);
                    else if (a.x_batch > 0) load_3d<CG>(el, dst, &maps.x, bar, kb * BK, 0, t0);
                    else load_2d<CG>(el, dst, k2 < 0 ? &maps.x : &maps.x2, bar, (k2 < 0 ? kb : k2) * BK, j0);
                }
                ++issued;
                if (++s == STAGES) { s = 0; par ^= 1; }
            }
        }
        if (failed && lane == 0) {
            status_raise(a.status, a.gen, PIMB200_ERR_TIMEOUT);
            // let the copies already issued land before the CTA gives its shared memory back (the leader's barriers count
            // them; the others wait for it below)
            if (counts)
                for (uint32_t q = issued > STAGES ? issued - STAGES : 0; q < issued; ++q)
                    for (uint32_t i = 0; i < (1u << 20); ++i)
                        if (mbar_try_wait(full0 + 8 * (q % STAGES), (q / STAGES) & 1)) break;
        }
    } else if (warp == 2) {
        // ---------------- MMA issuer (the pair's leader) ----------------
        if (rank == 0) {
            const uint32_t el = elect_one();
            // D = f32, A = B = f16, both K-major, N = bn, M = 128 or 256
            const uint32_t idesc = (1u << 4) | ((uint32_t)(a.bn >> 3) << 17) | ((uint32_t)(CG * BM >> 4) << 24);
            const uint64_t desc0 = make_smem_desc(smem_u32(smem));
            uint32_t s = 0, par = 0;
            int local = 0;
            for (int tile = first; tile < tiles && !failed; tile += stride, ++local) {
                const int as = local & 1;
                if (!mbar_wait(acce0 + 8 * as, ((uint32_t)(local >> 1) & 1) ^ 1, abort_flag, a.gen)) { failed = true; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d_tmem = tmem_base + (uint32_t)(as * BN);
                for (int k0 = 0; k0 < kblocks; k0 += KS) {
                    if (!mbar_wait(full0 + 8 * s, par, abort_flag, a.gen)) { failed = true; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < KS; ++i) {
                        if (i > 0 && k0 + i >= kblocks) break;
                        // descriptors count in 16-byte units: 16 halves inside the swizzle row are +2
                        const uint64_t adesc = desc0 + (uint64_t)((s * STAGE_BYTES + i * BLOCK_BYTES) >> 4), bdesc = adesc + (A_BYTES >> 4);
#pragma unroll
                        for (int k = 0; k < BK / UMMA_K; ++k)
                            mma<CG>(el, d_tmem, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc, (k0 > 0 || i > 0 || k > 0) ? 1u : 0u);
                    }
                    commit<CG>(el, empty0 + 8 * s);
                    if (++s == STAGES) { s = 0; par ^= 1; }
                }
                commit<CG>(el, accf0 + 8 * as);
            }
            if (failed) {
                if (lane == 0) status_raise(a.status, a.gen, PIMB200_ERR_TIMEOUT);
                __syncwarp();
                commit<CG>(el, accf0);             // wake the epilogue warps; they see the status word and leave
                commit<CG>(el, accf0 + 8);
            }
        }
    } else {
        // ---------------- epilogue: TMEM lane quarter = warp % 4, column half = every second chunk ----------------
        const int q = warp & 3, half = (warp - FIRST_EPI) >> 2;
        const int r = q * 32 + lane;                                   // row of the tile
        const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16);
        unsigned char* stg = staging + (warp - FIRST_EPI) * 2 * CHUNK_BYTES;   // this warp's two chunks
        int chunks = 0;                                                // chunks stored so far: selects the staging buffer
        const int rows_left = a.jrows - q * 32;                        // rows of this warp that belong to the tile
        const float lo = a.act == PIMB200_ACT_RELU ? 0.f : -INFINITY;
        int local = 0;
        for (int tile = first; tile < tiles; tile += stride, ++local) {
            const int as = local & 1;
            const int nt = tile % a.n_tiles;
            const int n0 = nt * a.bn, n_end = min(a.N, n0 + a.bn), j0 = ((tile / a.n_tiles) * CG + rank) * a.jrows, j = j0 + r;
            if (!mbar_wait(accf0 + 8 * as, (uint32_t)(local >> 1) & 1, abort_flag, a.gen)) {
                status_raise(a.status, a.gen, PIMB200_ERR_TIMEOUT);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = lane_base + (uint32_t)(as * BN);
            const bool row_ok = r < a.jrows && j < a.J;
            const uint4* bias4 = reinterpret_cast<const uint4*>(a.bias + n0);       // 8 at a time when none is past the end
            const bool bias_vec = a.bias && n0 + BN <= a.N && (reinterpret_cast<uintptr_t>(a.bias) & 15) == 0;
            if constexpr (EPI == kRowsHalf || EPI == kRowsFloat) {
                constexpr int CH = EPI == kRowsHalf ? 64 : 32;         // columns per 128-byte chunk
#pragma unroll 1
                for (int c = half * CH; c < BN; c += 2 * CH) {
                    if (n0 + c >= n_end) break;                        // uniform
                    uint4 bb[CH / 8];                                  // under way while the accumulator is read
                    if (bias_vec) {
#pragma unroll
                        for (int i = 0; i < CH / 8; ++i) bb[i] = ld_v4(bias4 + c / 8 + i);
                    }
                    uint32_t v[CH];
                    tmem_ld32_nowait(acc + (uint32_t)c, v);
                    if (CH == 64) tmem_ld32_nowait(acc + (uint32_t)c + 32, v + CH - 32);
                    tmem_wait_ld();
                    float f[CH];
#pragma unroll
                    for (int i = 0; i < CH; ++i) f[i] = __uint_as_float(v[i]);
                    if (bias_vec) {
#pragma unroll
                        for (int i = 0; i < CH / 8; ++i) {
                            float b[8];
                            widen8(bb[i], b);
#pragma unroll
                            for (int e = 0; e < 8; ++e) f[8 * i + e] += b[e];
                        }
                    } else if (a.bias) {
#pragma unroll
                        for (int i = 0; i < CH; ++i) f[i] += (n0 + c + i < n_end) ? __half2float(a.bias[n0 + c + i]) : 0.f;
                    }
                    uint4 o[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        if (EPI == kRowsHalf) {
                            const float* g = f + (8 * i) % CH;
                            o[i] = make_uint4(pack2(max_nan(g[0], lo), max_nan(g[1], lo)), pack2(max_nan(g[2], lo), max_nan(g[3], lo)),
                                              pack2(max_nan(g[4 % CH], lo), max_nan(g[5 % CH], lo)), pack2(max_nan(g[6 % CH], lo), max_nan(g[7 % CH], lo)));
                        } else {
                            o[i] = make_uint4(__float_as_uint(max_nan(f[4 * i], lo)), __float_as_uint(max_nan(f[4 * i + 1], lo)),
                                              __float_as_uint(max_nan(f[4 * i + 2], lo)), __float_as_uint(max_nan(f[4 * i + 3], lo)));
                        }
                    }
                    if (a.direct) {
                        // rows of Y that no tensor map takes: through shared memory too, but stored by the warp, a row at a time (a
                        // thread's own stores touch 32 rows at once: 656 rows of 8823 x 128 took 75 us)
                        unsigned char* buf = stg + (chunks & 1) * CHUNK_BYTES;
                        uint4* row = reinterpret_cast<uint4*>(buf + lane * 128);
#pragma unroll
                        for (int i = 0; i < 8; ++i) row[i ^ (lane & 7)] = o[i];
                        __syncwarp();
                        const int cols = min(CH, n_end - n0 - c), first_row = j0 + q * 32, rows = min(min(32, rows_left), a.J - first_row);
                        store_rows<EPI == kRowsFloat>(buf, a.Y, (size_t)first_row * a.ldy + n0 + c, a.ldy, rows, cols, a.direct == 2);
                        ++chunks;
                        continue;
                    }
                    if (n0 + c + CH > n_end && n_end < a.N) {          // half a chunk left of this tile: the map's boxes are whole ones
                        if (row_ok) {
                            unsigned char* yp = static_cast<unsigned char*>(a.Y) + ((size_t)j * a.ldy + n0 + c) * (EPI == kRowsHalf ? 2 : 4);
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                if (n0 + c + (i + 1) * CH / 8 <= n_end) reinterpret_cast<uint4*>(yp)[i] = o[i];
                        }
                        __syncwarp();
                        continue;
                    }
                    // the chunk before the previous one must have been read out of this buffer
                    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                    __syncwarp();
                    unsigned char* buf = stg + (chunks & 1) * CHUNK_BYTES;
                    uint4* row = reinterpret_cast<uint4*>(buf + lane * 128);
#pragma unroll
                    for (int i = 0; i < 8; ++i) row[i ^ (lane & 7)] = o[i];   // the 128-byte swizzle of the store's map
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        if (rows_left >= 32) tma_store_2d(&maps.y, smem_u32(buf), n0 + c, j0 + q * 32);
                        else if (rows_left > 0) tma_store_2d(&maps.y_tail, smem_u32(buf), n0 + c, j0 + q * 32);
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                    ++chunks;
                }
            } else if constexpr (EPI == kRowsArgmax) {
                // values are rounded to fp16 first, as the stored logits would be; ascending columns and a strict
                // comparison keep the lowest index among equal maxima
                float bv = -INFINITY;
                int bi = n0 + half * 32;
#pragma unroll 1
                for (int c = half * 32; c < BN; c += 64) {
                    const int nb = n0 + c;
                    if (nb >= n_end) break;
                    uint4 bb[4];
                    if (bias_vec) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) bb[i] = ld_v4(bias4 + c / 8 + i);
                    }
                    uint32_t v[32];
                    tmem_ld32(acc + (uint32_t)c, v);
                    const int lim = n_end - nb;
                    float b[32];
                    if (bias_vec) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) widen8(bb[i], b + 8 * i);
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i) b[i] = (a.bias && i < lim) ? __half2float(a.bias[nb + i]) : 0.f;
                    }
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const float f = __half2float(__float2half_rn(__uint_as_float(v[i]) + b[i]));
                        if (f > bv && i < lim) { bv = f; bi = nb + i; }
                    }
                }
                if (row_ok) {
                    const size_t at = (size_t)(2 * nt + half) * a.J + j;
                    a.best_v[at] = bv;
                    a.best_i[at] = bi;
                }
            } else {
                // LSTM cell: 64 columns = the four gates (i, f, g, o side by side) of 16 hidden units
#pragma unroll 1
                for (int c = half * 64; c < BN; c += 128) {
                    if (n0 + c >= n_end) break;
                    uint32_t v[64];
                    tmem_ld32_nowait(acc + (uint32_t)c, v);
                    tmem_ld32_nowait(acc + (uint32_t)c + 32, v + 32);
                    tmem_wait_ld();
                    if (row_ok) {
                    const int u0 = (n0 + c) >> 2;
                    float cp[16], hv[16];
                    if (a.c0) load_half16(a.c0 + (size_t)j * a.H + u0, cp);
                    else {
#pragma unroll
                        for (int i = 0; i < 16; ++i) cp[i] = 0.f;
                    }
                    const float4* b4 = reinterpret_cast<const float4*>(a.cell_bias) + u0;
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float4 b = __ldg(b4 + i);        // (a constant of the handle)
                        const float zi = __uint_as_float(v[4 * i]) + b.x, zf = __uint_as_float(v[4 * i + 1]) + b.y,
                                    zg = __uint_as_float(v[4 * i + 2]) + b.z, zo = __uint_as_float(v[4 * i + 3]) + b.w;
                        cp[i] = sigmoidf_(zf) * cp[i] + sigmoidf_(zi) * tanhf_(zg);
                        hv[i] = __half2float(__float2half_rn(sigmoidf_(zo) * tanhf_(cp[i])));
                    }
                    uint32_t w[8];
                    if (a.cn) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) w[i] = pack2(cp[2 * i], cp[2 * i + 1]);
                        store_half16(a.cn + (size_t)j * a.H + u0, w);
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) w[i] = pack2(hv[2 * i], hv[2 * i + 1]);
                    if (a.hn) store_half16(a.hn + (size_t)j * a.H + u0, w);
                    if (a.res) {
                        float rv[16];
                        load_half16(a.res + (size_t)j * a.res_ld + u0, rv);
#pragma unroll
                        for (int i = 0; i < 8; ++i) w[i] = pack2(hv[2 * i] + rv[2 * i], hv[2 * i + 1] + rv[2 * i + 1]);
                    }
                    store_half16(a.y + (size_t)j * a.y_ld + u0, w);
                    }
                    __syncwarp();                                      // the next chunk's TMEM load is warp-wide
                }
            }
            // this warp is done reading the stage: hand it back to the MMA issuer.  Only TMEM reads are ordered by this, and
            // those are complete: a release would wait for the warp's output stores (2500 cycles a tile)
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                if (CG == 1) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acce0 + 8 * as) : "memory");
                else asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(mapa(acce0 + 8 * as, 0)) : "memory");
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the staging rows have been read
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    pair_sync<CG>();                               // neither CTA leaves while the other may still signal it
    if (warp == 2) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (CG == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS) : "memory");
    }
}

// ---- host side ---------------------------------------------------------------------------------
namespace {

constexpr int kMaxDevices = 64;

template <int BN, int EPI, int CG>
int launch_one(const Maps& m, const Args& a, int dev, cudaStream_t st) {
    static bool attr_set[kMaxDevices];   // cudaFuncSetAttribute is per device
    constexpr size_t smem = smem_for(BN, CG);
    if (!attr_set[dev]) {
        PIMB200_CUDA_TRY(cudaFuncSetAttribute(gemm_rows_kernel<BN, EPI, CG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set[dev] = true;
    }
    const long tiles = (long)a.j_tiles * a.n_tiles;
    const int slots = tc_sm_count(dev) / CG, grid = CG * (int)(tiles < slots ? tiles : slots);
    return cuda_status(launch_pdl<CG>(gemm_rows_kernel<BN, EPI, CG>, dim3(grid), dim3(THREADS), smem, st, m, a));
}

struct Plan { int bn, cg; };       // weight rows per tile, CTAs per tile

// Tile shape.  For one, two, ... waves of tiles over the SMs (or pairs of them) the tiles are made as narrow as those waves
// allow, so that no wave is left half empty (32320 weight rows: 145 tiles of 224 on 148 SMs, not 127 of 256).  A wave takes
// as long as the slower of its K blocks and its epilogue; the last epilogue comes on top, nothing hides it.  Cycles per K
// block of 64 as measured (single CTAs of 64 / 128 / 256 columns: 300 / 400 / 700, pairs 320 / 400 / 520: MMAs where they
// bound, operand traffic or barrier waits where those do).  One wave of short products is quickest with single CTAs, many
// waves with pairs of 256 columns (also where the epilogue is all that counts: 128000 rows of 4096 x 240 take 470 us with
// single CTAs, 429 with pairs).
Plan pick(int N, int J, int jrows, int kblocks, int grain, int sms) {
    static const int per_block[2][3] = {{300, 400, 700}, {320, 400, 520}};
    Plan best{0, 0};
    double cost = 0;
    for (int cg = J > jrows ? 2 : 1; cg >= 1; --cg) {
        const int slots = sms / cg, j_tiles = ceil_div(J, jrows * cg);
        int last = 0;
        for (long w = (long)ceil_div(N, 256) * j_tiles / slots; ; ++w) {
            const long n_max = w * slots / j_tiles;                    // column tiles that w waves hold
            if (n_max < 1) continue;
            int bn = (int)((N + n_max - 1) / n_max);
            bn = ceil_div(bn, grain) * grain;
            if (bn > 256) continue;
            if (bn < 64) bn = 64;
            if (bn == last) break;
            last = bn;
            const long tiles = (long)j_tiles * ceil_div(N, bn), waves = (tiles + slots - 1) / slots;
            const int* p = per_block[cg - 1];
            const double per = bn <= 128 ? p[0] + (p[1] - p[0]) * (bn - 64) / 64.0 : p[1] + (p[2] - p[1]) * (bn - 128) / 128.0;
            const double mma = kblocks * per, epi = 600 + 14 * bn;
            const double c = waves * (300 + (mma > epi ? mma : epi)) + epi;
            if (!best.bn || c < cost) { best = Plan{bn, cg}; cost = c; }
            if (bn == 64) break;
        }
    }
    return best;
}

template <int EPI>
int launch_plan(Plan p, const Maps& m, Args& a, int dev, cudaStream_t st) {
    a.bn = p.bn;
    a.n_tiles = ceil_div(a.N, p.bn);
    a.j_tiles = ceil_div(a.J, a.jrows * p.cg);
    if (p.cg == 2) {
        if (p.bn > 128) return launch_one<256, EPI, 2>(m, a, dev, st);
        return p.bn > 64 ? launch_one<128, EPI, 2>(m, a, dev, st) : launch_one<64, EPI, 2>(m, a, dev, st);
    }
    if (p.bn > 128) return launch_one<256, EPI, 1>(m, a, dev, st);
    return p.bn > 64 ? launch_one<128, EPI, 1>(m, a, dev, st) : launch_one<64, EPI, 1>(m, a, dev, st);
}

int tile_rows(int J) { return J < BM ? J : BM; }

bool operands_ok(const void* W, const void* X, int K, long ldx) {
    return K % 8 == 0 && ldx % 8 == 0 && aligned16(W) && aligned16(X);
}

}  // namespace
}  // namespace tc

int launch_gemm_rows(const __half* W, const __half* X, const __half* bias, void* Y, int N, int K, int J, int ldx, int ldy,
                     int act, int y_is_f32, int x_batch, long x_seq_rows, cudaStream_t st, int fixed) {
    using namespace tc;
    if (!operands_ok(W, X, K, ldx)) return PIMB200_ERR_UNSUPPORTED;
    if (x_batch > 0 && (J % x_batch != 0 || x_batch > BM)) return PIMB200_ERR_UNSUPPORTED;
    Args a = {};
    int dev = 0, rc;
    if ((rc = tc_prepare(&dev, &a.status, &a.gen)) != PIMB200_OK) return rc;
    a.bias = bias; a.N = N; a.J = J; a.act = act; a.fixed = fixed;
    // whole timesteps, or no more rows than there are: a tile's other rows are never stored, and a load of rows past the end
    // of X costs more than one of rows that exist (32320 x 1024, 32 rows: 19.2 us with boxes of 128)
    a.jrows = x_batch > 0 ? BM / x_batch * x_batch : tile_rows(J);
    a.x_batch = x_batch;
    a.kb1 = ceil_div(K, BK);
    const Plan p = pick(N, J, a.jrows, a.kb1, 32, tc_sm_count(dev));
    Maps m = {};
    if (!encode_2d(&m.w, W, N, K, (uint64_t)K * 2, p.bn / p.cg, 2)) return PIMB200_ERR_UNSUPPORTED;
    if (x_batch > 0) {
        if (!encode_x_time_major(&m.x, X, x_batch, J / x_batch, x_seq_rows, K, (uint64_t)ldx * 2, a.jrows / x_batch))
            return PIMB200_ERR_UNSUPPORTED;
    } else if (!encode_2d(&m.x, X, J, K, (uint64_t)ldx * 2, a.jrows, 2)) {
        return PIMB200_ERR_UNSUPPORTED;
    }
    const int es = y_is_f32 ? 4 : 2, tail = a.jrows % 32, whole = a.jrows < 32 ? a.jrows : 32;
    a.Y = Y; a.ldy = ldy;
    // (a store through a map writes whole 16 bytes: the last of a row of another width would reach into what lies behind it)
    a.direct = !aligned16(Y) || ((long)ldy * es | (long)N * es) % 16 != 0;
    if (a.direct && ((long)ldy * es | (long)(reinterpret_cast<uintptr_t>(Y))) % 4 == 0) a.direct = 2;
    if (a.direct) m.y = m.x;   // (prefetched only)
    else if (!encode_2d(&m.y, Y, J, N, (uint64_t)ldy * es, whole, es) ||
        (tail && !encode_2d(&m.y_tail, Y, J, N, (uint64_t)ldy * es, tail, es)))
        return PIMB200_ERR_UNSUPPORTED;
    return y_is_f32 ? launch_plan<kRowsFloat>(p, m, a, dev, st) : launch_plan<kRowsHalf>(p, m, a, dev, st);
}

int gemm_rows_max_parts(int N) { return 2 * ceil_div(N, 64); }

int launch_gemm_rows_argmax(const __half* W, const __half* X, const __half* bias, float* best_v, int* best_i, int* parts, int N,
                            int K, int J, int ldx, cudaStream_t st) {
    using namespace tc;
    if (!operands_ok(W, X, K, ldx)) return PIMB200_ERR_UNSUPPORTED;
    Args a = {};
    int dev = 0, rc;
    if ((rc = tc_prepare(&dev, &a.status, &a.gen)) != PIMB200_OK) return rc;
    a.bias = bias; a.N = N; a.J = J; a.act = PIMB200_ACT_NONE;
    a.jrows = tile_rows(J);
    a.kb1 = ceil_div(K, BK);
    const Plan p = pick(N, J, a.jrows, a.kb1, 32, tc_sm_count(dev));
    *parts = 2 * ceil_div(N, p.bn);
    a.best_v = best_v; a.best_i = best_i;
    Maps m = {};   // (y is only prefetched)
    if (!encode_2d(&m.w, W, N, K, (uint64_t)K * 2, p.bn / p.cg, 2) || !encode_2d(&m.x, X, J, K, (uint64_t)ldx * 2, a.jrows, 2))
        return PIMB200_ERR_UNSUPPORTED;
    m.y = m.x;
    return launch_plan<kRowsArgmax>(p, m, a, dev, st);
}

int launch_gemm_rows_cell(const RowsCell& c, cudaStream_t st) {
    using namespace tc;
    if (c.H % 16 != 0 || !operands_ok(c.Wx, c.x, c.I, c.x_ld) || (c.h0 && !operands_ok(c.Wh, c.h0, c.H, c.H)) ||
        (c.c0 && !aligned16(c.c0)) || !aligned16(c.y) || c.y_ld % 8 != 0 || (c.hn && !aligned16(c.hn)) ||
        (c.cn && !aligned16(c.cn)) || (c.res && (!aligned16(c.res) || c.res_ld % 8 != 0)))
        return PIMB200_ERR_UNSUPPORTED;
    Args a = {};
    int dev = 0, rc;
    if ((rc = tc_prepare(&dev, &a.status, &a.gen)) != PIMB200_OK) return rc;
    a.N = 4 * c.H; a.J = c.J; a.jrows = tile_rows(c.J); a.fixed = 1;
    a.kb1 = ceil_div(c.I, BK);
    a.kb2 = c.h0 ? ceil_div(c.H, BK) : 0;
    a.cell_bias = c.bias; a.c0 = c.c0; a.y = c.y; a.y_ld = c.y_ld; a.hn = c.hn; a.cn = c.cn; a.res = c.res; a.res_ld = c.res_ld;
    a.H = c.H;
    const Plan p = pick(a.N, a.J, a.jrows, a.kb1 + a.kb2, 64, tc_sm_count(dev));
    Maps m = {};
    if (!encode_2d(&m.w, c.Wx, a.N, c.I, (uint64_t)c.I * 2, p.bn / p.cg, 2) ||
        !encode_2d(&m.x, c.x, c.J, c.I, (uint64_t)c.x_ld * 2, a.jrows, 2))
        return PIMB200_ERR_UNSUPPORTED;
    if (c.h0 && (!encode_2d(&m.w2, c.Wh, a.N, c.H, (uint64_t)c.H * 2, p.bn / p.cg, 2) ||
                 !encode_2d(&m.x2, c.h0, c.J, c.H, (uint64_t)c.H * 2, a.jrows, 2)))
        return PIMB200_ERR_UNSUPPORTED;
    m.y = m.x;
    return launch_plan<kRowsCell>(p, m, a, dev, st);
}

}  // namespace pimb200
