// Convolutions on the tensor cores as windows over an image (implicit GEMM): the transposed convolution of coefficient
// rows (CROWN backward), the attack's and the optimisation's forward and gradient convolutions.  For every
// output pixel, out[n] = sum over taps and channels of in[pixel shifted by the tap][c] * W[tap][c][n].
//
// What it replaces wrote the products of every pixel with every tap to memory and gathered them again (a residual layer
// of 64 channels on 32 x 32 pixels and 4608 rows: 10.9 GB written and read per layer, 7 ms).  Here a CTA loads the halo of
// an 8 x 16 pixel tile once, and every tap is the same shared-memory tile read from another start address: pixels are
// rows of 32, 64 or 128 bytes of channels in a swizzled layout whose pattern depends on the address alone, a tile's
// sixteen groups of eight pixels are a constant distance apart, so a shifted window is one operand descriptor.  The
// layer's weights stay in shared memory for the whole launch; DRAM sees the input once (halo overlap in L2) and the
// output once.
//
// Arithmetic: three products of split operands, a = 2^-s (ah + 2^-11 al) with fp16 parts of 11 bits each (kind::f16 runs
// at twice the rate of kind::tf32 and moves half the bytes; a TF32 pair has the same 22 bits).  Rows and weights are
// scaled by powers of two so that their largest magnitude lies in [2^14, 2^15).  Ah*Wh goes into a MAIN accumulator that is
// drained into fp32 registers every few steps, Al*Wh + Ah*Wl into a CROSS accumulator added once at the end.
// Rounding (win_eps): operand split 0.75 * 2^-20 as for a TF32 pair; each MMA step at most one fp32 ulp of the
// accumulated magnitude (the model of k_umma_tf32x3; element by element in tests/test_gpu_rates.py); one fp32 addition per chain.  An element
// more than 2^29 times smaller than its row's largest loses its low bits to fp16's exponent range: an absolute error of
// at most 2^-50 of that largest magnitude, which k_split_image charges to the row separately; weights that small
// make a layer ineligible (win_prepare gets a negative wmax).
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "nyb200_internal.cuh"
#include "nyb200_tcgen05.cuh"

namespace nyb {

namespace win {

constexpr int TX = 8, TY = 16;            // output pixels of a tile: 128 rows of the product
constexpr int MAXS = 16, MAXT = 64;       // input sources, taps
constexpr int EPI_GROUPS = 2;             // epilogue groups of four warps, up to 32 columns each
constexpr int THREADS = 128 + EPI_GROUPS * 128;
constexpr int SMEM_MOST = 226 * 1024;

struct Source { int dy, dx, ntaps, tap0, tw; };   // first halo row / column relative to the tile; its taps, tw in a row

struct Params {
    int rows, Cp, sw, swa, nchunk, Nb, N, n_blocks;   // channels padded, bytes of a weight row and of a pixel row in shared memory,
                                                 // 64-channel chunks, output columns
    int n_src, taps, tpc, chains, in_step, s;    // taps per MAIN chain, chains per tile; input stride; output parities per axis
    int out_c, out_h, out_w, out_plane, exact, pair;
    int bx, by, tiles_y, tiles_x;                // halo box, tiles of a row
    int slot_bytes, slots, w_tile_bytes;
    Source src[MAXS];
    const float *row_inv;                        // [rows] scale of the row, undone; null: 1
    float w_inv;
    float *out;
    long ldo;
    int pixel_major;                             // the channels of a result's pixel together, not its planes
    unsigned *row_max;                           // largest magnitude of a result's row (bits), or null
    int *err;
};

}  // namespace win

using namespace umma;
using namespace win;

// Roles: warp 0 loads halo tiles, warps 1 and 3 issue the products, warp 2 owns the tensor memory, the other eight warps are
// two epilogue groups of up to 32 columns each: a tile of 64 columns is drained by both at once, narrower tiles go to them in
// turn (a small layer's tile is a few dozen products; its way through the barriers and tensor memory is longer than they take).
// Per tile: warp 3 adds Al*Wh and Ah*Wl over all taps into the tile's CROSS columns, warp 1 Ah*Wh in chains, each into MAIN
// columns of its own.  Up to 32 channels the high and low parts share a pixel's row (one load); from 64 on they are two tiles,
// and the low one is free for the next loads after its pass.
// The ring: a wait on a barrier tells the phase it is for from the ones next to it, no more, so nobody may get two phases away from
// a barrier it waits on.  A slot's b_full is completed by its load alone, and the next load waits for two arrivals at b_empty,
// one of each issuing warp, each after that warp's own wait on this b_full: b_full's next phase begins behind both waits, and
// b_empty's behind the loads' thread's.  That holds for low tiles too, which warp 1 does not read: were it to pass them by, a low
// tile that is late (the slots' number may be odd: a slot then holds low and high tiles in turn) would leave b_full where the
// high tile after it is waited for, and the low one, or half of it, would be multiplied in its place.
// What bounds it: shared memory, at three quarters of its rate.  A 128 x 64 x 16 product takes 48 cycles (its operands' bytes),
// so a tile of 64 columns, 9 taps and 64 channels 5.2 thousand.  From one warp, whose loop the compiler took for divergent, with
// [Wh | Wl] as one product of 128 columns (4.0 thousand), a tile took 12.2 thousand; with converged loops (mbar_wait_warp) 9.7;
// from two warps with 64-column products, which halve what the epilogue drains and double its buffers, 8.5; with eight epilogue
// warps instead of sixteen, results pixel-major where the next pass wants them so (the stores were 3.7 thousand of it) and the
// warp's number shuffled, so that the compiler knows it uniform, 7.1 (7.3 since both issuing warps follow every slot of the ring).
// All products from one warp: 9.5.
template <int KS, int NB>
__global__ void __launch_bounds__(win::THREADS, 1)
k_conv_win(const __grid_constant__ CUtensorMap tm_hi, const __grid_constant__ CUtensorMap tm_lo, const __grid_constant__ CUtensorMap tm_w,
           const __grid_constant__ Params P) {
    constexpr bool PACK = KS < 4;
    constexpr int GC = NB >= 32 ? 32 : 16, CS = NB / GC, TG = EPI_GROUPS / CS;   // columns of a group, column groups, tile groups
    constexpr int MAIN_BUFS = NB == 64 ? 6 : NB == 32 ? 10 : 16, CROSS_BUFS = NB == 64 ? 2 : NB == 32 ? 6 : 8;
    static_assert((MAIN_BUFS + CROSS_BUFS) * NB <= 512, "tensor memory columns");
    static_assert(CROSS_BUFS % TG == 0, "a cross buffer and its tile-start barrier belong to one group");
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int w_tiles = P.taps * P.nchunk * 2;
    unsigned char *wbase = smem, *ring = smem + (size_t)w_tiles * P.w_tile_bytes;
    unsigned long long *bars = (unsigned long long *)(ring + (size_t)P.slots * P.slot_bytes);
    unsigned long long *b_full = bars, *b_empty = bars + P.slots, *b_mf = b_empty + P.slots, *b_me = b_mf + MAIN_BUFS,
                       *b_cf = b_me + MAIN_BUFS, *b_ce = b_cf + CROSS_BUFS, *b_ts = b_ce + CROSS_BUFS, *b_w = b_ts + CROSS_BUFS;
    unsigned *tmem_slot = (unsigned *)(b_w + 1);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
    int *col_off = (int *)(tmem_slot + 2);        // [NB] output offset of a column; parities of a column behind it
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;   // (the same in a warp, as the compiler sees it too)
    const int n_block = blockIdx.x % P.n_blocks;
    pdl_trigger();
    if (threadIdx.x == 0) {
        for (int s = 0; s < P.slots; ++s) { mbar_init(smem_u32(&b_full[s]), 1); mbar_init(smem_u32(&b_empty[s]), 2); }
        for (int b = 0; b < MAIN_BUFS; ++b) { mbar_init(smem_u32(&b_mf[b]), 1); mbar_init(smem_u32(&b_me[b]), 4 * CS); }
        for (int b = 0; b < CROSS_BUFS; ++b) { mbar_init(smem_u32(&b_cf[b]), 1); mbar_init(smem_u32(&b_ce[b]), 4 * CS); mbar_init(smem_u32(&b_ts[b]), 1); }
        mbar_init(smem_u32(b_w), 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int j = threadIdx.x; j < NB; j += win::THREADS) {
        const int n = n_block * NB + j, px = n % P.s, c = (n / P.s) % P.out_c, py = n / (P.s * P.out_c);
        col_off[j] = c * P.out_plane + py * P.out_w + px;
        col_off[NB + j] = py * 16 + px;
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    pdl_wait();
    const unsigned tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    // this CTA's tiles t0, t0 + tstep, ...: fewer than 2^31 of them in all (launch_win)
    const int per_row = P.tiles_y * P.tiles_x, tiles = P.rows * per_row, t0 = blockIdx.x / P.n_blocks, tstep = gridDim.x / P.n_blocks;

    if (warp < 4) {
        if (warp == 0 && lane == 0) {
            // ------------------------------------------------------------ loads
            mbar_expect_tx(smem_u32(b_w), (unsigned)(w_tiles * P.w_tile_bytes));
            for (int i = 0; i < w_tiles; ++i) {   // tile (tap, chunk, part): columns chunk * 64, rows of the part's block
                const int part = i & 1, tc = i >> 1, tap = tc / P.nchunk, ch = tc - tap * P.nchunk;
                tma_load_2d(smem_u32(wbase + (size_t)i * P.w_tile_bytes), &tm_w, ch * 64, ((part * P.taps + tap) * P.n_blocks + n_block) * NB, smem_u32(b_w));
            }
            int sl = 0;
            unsigned ph = 1;
            for (int t = t0; t < tiles && !*abort_flag; t += tstep) {
                const int row = t / per_row, r = t - row * per_row, ty = r / P.tiles_x, tx = r - ty * P.tiles_x;
                for (int s = 0; s < P.n_src; ++s) {
                    const int y = ty * TY * P.in_step + P.src[s].dy, x = tx * TX * P.in_step + P.src[s].dx;
                    for (int ch = 0; ch < P.nchunk; ++ch)
                        for (int part = PACK ? 1 : 0; part < 2; ++part) {   // low parts first
                            if (!mbar_wait_soon(smem_u32(&b_empty[sl]), ph)) { atomicExch(P.err, 21); *abort_flag = 1; goto done_load; }
                            mbar_expect_tx(smem_u32(&b_full[sl]), (unsigned)(P.bx * P.by * P.swa));
                            tma_load_4d(smem_u32(ring + (size_t)sl * P.slot_bytes), part ? &tm_hi : &tm_lo, ch * 64, x, y, row, smem_u32(&b_full[sl]));
                            if (++sl == P.slots) { sl = 0; ph ^= 1; }
                        }
                }
            }
        done_load:;
        } else if (warp == 1 || warp == 3) {
            // ------------------------------------------------------------ products: warp 3 the cross terms, warp 1 the chains
            const bool cross = warp == 3;
            const unsigned idesc = make_idesc_f16(128, NB);
            // a descriptor is its constant upper word and the start address in 16-byte units plus the fixed bit 16
            const unsigned a_hi = (unsigned)(make_desc_sw(0, P.swa, (unsigned)(P.bx * P.swa)) >> 32), w_hi = (unsigned)(make_desc_sw(0, P.sw, (unsigned)(8 * P.sw)) >> 32);
            const unsigned w_lo0 = ((smem_u32(wbase) & 0x3FFFF) >> 4) | (1u << 16), w_part = (unsigned)P.w_tile_bytes >> 4, w_chunk = 2 * w_part,
                           w_tap = (unsigned)P.nchunk * w_chunk;
            auto desc = [](unsigned hi, unsigned lo) { return ((unsigned long long)hi << 32) | lo; };
            const unsigned px = (unsigned)P.swa >> 4;   // from a tap's pixels to the next one's
            auto fail = [&](int code) { if (lane == 0) { atomicExch(P.err, code); *abort_flag = 1; } };
            bool ok = mbar_wait_warp(smem_u32(b_w), 0);
            if (!ok) fail(22);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            int sl = 0, mbuf = 0, cb = 0;
            unsigned ph = 0, mph = 1, cph = 1;
            auto next_slot = [&]() { if (++sl == P.slots) { sl = 0; ph ^= 1; } };
            for (int t = t0; t < tiles && ok && !flag_warp(abort_flag); t += tstep) {
                // (warp 1 too, for b_ts below)
                if (!mbar_wait_warp(smem_u32(&b_ce[cb]), cph)) { fail(23); break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned d_cross = tmem_base + (unsigned)((MAIN_BUFS + cb) * NB);
                unsigned on = 0;
                bool begun = false;
                for (int s = 0; s < P.n_src && ok; ++s) {
                    const int nt = P.src[s].ntaps, tap0 = P.src[s].tap0, tw = P.src[s].tw;
                    const unsigned row_step = (unsigned)(P.bx - tw) * px;   // further, to the next row's first tap
                    for (int ch = 0; ch < P.nchunk; ++ch) {
                        const unsigned w0 = w_lo0 + tap0 * w_tap + ch * w_chunk;
                        // the pixels' parts in the slot (a) times the weights' part (w), tap by tap, into the cross accumulator
                        auto cross_pass = [&](unsigned a, unsigned w) {
                            for (int tap = 0, tx = 0; tap < nt; ++tap) {
                                mma_f16_group<KS>(d_cross, desc(a_hi, a), desc(w_hi, w), idesc, on);
                                on = 1;
                                w += w_tap;
                                a += px;
                                if (++tx == tw) { tx = 0; a += row_step; }
                            }
                        };
                        auto start_of_slot = [&]() { return (((smem_u32(ring) + (unsigned)(sl * P.slot_bytes)) & 0x3FFFF) >> 4) | (1u << 16); };
                        if (!PACK) {
                            // The low parts' tile: the cross warp's data alone, but both warps wait for it and both release it (see
                            // the ring, above)
                            if (!mbar_wait_warp(smem_u32(&b_full[sl]), ph)) { fail(24); ok = false; break; }
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            if (cross) {
                                cross_pass(start_of_slot(), w0);
                                mma_commit_elect(smem_u32(&b_empty[sl]));
                            } else {
                                if (lane == 0) mbar_arrive(smem_u32(&b_empty[sl]));
                                __syncwarp();
                            }
                            next_slot();
                        }
                        if (!mbar_wait_warp(smem_u32(&b_full[sl]), ph)) { fail(25); ok = false; break; }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        unsigned a = start_of_slot(), w = w0;
                        if (cross) {
                            if (PACK) cross_pass(a + 2 * KS, w0);
                            cross_pass(a, w0 + w_part);
                        } else
                            for (int tap = 0, tx = 0; tap < nt;) {
                                if (!mbar_wait_warp(smem_u32(&b_me[mbuf]), mph)) { fail(26); ok = false; break; }
                                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                                // The tile's groups may look at its first buffer now: the buffer's previous use, perhaps other
                                // groups', is over.  (A barrier's parity only tells one use from the next; a group that
                                // waited two uses ahead would take the use before the last for its own.  The other buffers'
                                // previous uses end before this chain does: the chains complete in order.)  One barrier per cross
                                // buffer: its previous tile's groups have looked at it, since they have given that buffer back
                                // (b_ce).  Chains alone do not tell: tiles of one or two fit the buffers many times.
                                if (!begun) { if (lane == 0) mbar_arrive(smem_u32(&b_ts[cb])); __syncwarp(); begun = true; }
                                const unsigned d_main = tmem_base + (unsigned)(mbuf * NB);
                                const int end = min(nt, tap + P.tpc);
                                on = 0;
                                for (; tap < end; ++tap) {
                                    mma_f16_group<KS>(d_main, desc(a_hi, a), desc(w_hi, w), idesc, on);
                                    on = 1;
                                    w += w_tap;
                                    a += px;
                                    if (++tx == tw) { tx = 0; a += row_step; }
                                }
                                mma_commit_elect(smem_u32(&b_mf[mbuf]));
                                if (++mbuf == MAIN_BUFS) { mbuf = 0; mph ^= 1; }
                            }
                        if (!ok) break;
                        mma_commit_elect(smem_u32(&b_empty[sl]));
                        next_slot();
                    }
                }
                if (cross && ok) mma_commit_elect(smem_u32(&b_cf[cb]));
                if (++cb == CROSS_BUFS) { cb = 0; cph ^= 1; }
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue: thread = one pixel, GC columns
        const int q = warp & 3, group = (warp - 4) >> 2, tgroup = group / CS, col0 = (group % CS) * GC;
        const unsigned lane_base = tmem_base + ((unsigned)(q * 32) << 16);
        const int pr = q * 32 + lane, n_here = min(GC, P.N - n_block * NB - col0);
        unsigned mbuf = (unsigned)(tgroup * P.chains) % MAIN_BUFS, mph = ((unsigned)(tgroup * P.chains) / MAIN_BUFS) & 1;
        int cb = tgroup % CROSS_BUFS;
        unsigned cph = 0;
        // pixel-major results: sixteen columns of this thread are channels from n_first on, of one row parity where there are two
        int n_first[GC / 16], n_row[GC / 16];
#pragma unroll
        for (int h = 0; h < GC / 16; ++h) {
            const int n = n_block * NB + col0 + 16 * h;
            n_first[h] = P.s == 1 ? n : (n / 2) % P.out_c; n_row[h] = P.s == 1 ? 0 : n / (2 * P.out_c);
        }
        auto load = [&](unsigned from, unsigned (&r)[GC]) {
#pragma unroll
            for (int h = 0; h < GC / 16; ++h) tmem_ld16(lane_base + from + 16 * h, *(unsigned (*)[16])&r[16 * h]);
        };
        for (int t = t0 + tgroup * tstep; t < tiles; t += TG * tstep) {
            float sum[GC];
#pragma unroll
            for (int j = 0; j < GC; ++j) sum[j] = 0.f;
            // where the tile's results go, and the row's scale, on its way from memory while the products run
            const int row = t / per_row, rt = t - row * per_row, ty = rt / P.tiles_x, tx = rt - ty * P.tiles_x;
            const int y = (ty * TY + (pr >> 3)) * P.s, x = (tx * TX + (pr & 7)) * P.s;
            const float row_scale = P.row_inv ? __ldg(P.row_inv + row) : 1.f;
            bool ok = mbar_wait_warp(smem_u32(&b_ts[cb]), cph);
            if (!ok) { if (lane == 0) { atomicExch(P.err, 29); *abort_flag = 1; } break; }
            // two chains at a time: their loads out of tensor memory overlap
            for (int i = 0; i < P.chains && ok; i += 2) {
                const unsigned m0 = mbuf, ph0 = mph;
                if (++mbuf == MAIN_BUFS) { mbuf = 0; mph ^= 1; }
                const unsigned m1 = mbuf, ph1 = mph;
                const bool two = i + 1 < P.chains;
                if (two && ++mbuf == MAIN_BUFS) { mbuf = 0; mph ^= 1; }
                ok = mbar_wait_warp(smem_u32(&b_mf[m0]), ph0);
                if (!ok) { if (lane == 0) { atomicExch(P.err, 27); *abort_flag = 1; } break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                unsigned r[GC], r1[GC];
                load(m0 * NB + col0, r);
                if (two) {
                    ok = mbar_wait_warp(smem_u32(&b_mf[m1]), ph1);
                    if (!ok) { if (lane == 0) { atomicExch(P.err, 27); *abort_flag = 1; } break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    load(m1 * NB + col0, r1);
                }
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) { mbar_arrive(smem_u32(&b_me[m0])); if (two) mbar_arrive(smem_u32(&b_me[m1])); }
#pragma unroll
                for (int u = 0; u < GC; ++u) sum[u] += __uint_as_float(r[u]);
                if (two)
#pragma unroll
                    for (int u = 0; u < GC; ++u) sum[u] += __uint_as_float(r1[u]);
            }
            if (!ok) break;
            ok = mbar_wait_warp(smem_u32(&b_cf[cb]), cph);
            if (!ok) { if (lane == 0) { atomicExch(P.err, 28); *abort_flag = 1; } break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            {
                unsigned c[GC];
                load((MAIN_BUFS + cb) * NB + col0, c);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&b_ce[cb]));
#pragma unroll
                for (int u = 0; u < GC; ++u) sum[u] = fmaf(__uint_as_float(c[u]), 4.8828125e-4f /* 2^-11 */, sum[u]);
            }
            // the chains and the cross buffers of the other groups' tiles lie in between
            const unsigned skip = (unsigned)((TG - 1) * P.chains) + mbuf;
            mph ^= (skip / MAIN_BUFS) & 1;
            mbuf = skip % MAIN_BUFS;
            cb += TG;
            if (cb >= CROSS_BUFS) { cb -= CROSS_BUFS; cph ^= 1; }
            const float scale = row_scale * P.w_inv;
            const bool inside = y < P.out_h && x < P.out_w;
            if (P.row_max) {   // (columns past the last one are zero; so are, with even sides, the pixels past the image)
                float m = 0.f;
#pragma unroll
                for (int u = 0; u < GC; ++u) m = fmaxf(m, fabsf(sum[u]));
                // a NaN is none of its row's maxima: its products say so themselves
                const unsigned w = __reduce_max_sync(0xffffffffu, inside ? __float_as_uint(m * scale) : 0u);
                if (lane == 0 && w) atomicMax(P.row_max + row, w);
            }
            if (P.pixel_major) {
                float *o = P.out + (long)row * P.ldo;
                if (P.s == 1) {
                    // Sixteen channels of a pixel are 64 bytes.  Four lanes exchange theirs so that a store is eight runs of 64
                    // bytes and not 32 of 16 (the line looked up is what a store costs).
#pragma unroll
                    for (int h = 0; h < GC / 16; ++h) {
                        float4 q4[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            q4[k] = make_float4(sum[16 * h + 4 * k] * scale, sum[16 * h + 4 * k + 1] * scale, sum[16 * h + 4 * k + 2] * scale, sum[16 * h + 4 * k + 3] * scale);
                        auto swap4 = [&](float4 &lo4, float4 &hi4, int step) {   // this lane's part of a 2 x 2 transposition
                            const bool up = lane & step;
                            float4 v = up ? lo4 : hi4;
                            v.x = __shfl_xor_sync(0xffffffffu, v.x, step); v.y = __shfl_xor_sync(0xffffffffu, v.y, step);
                            v.z = __shfl_xor_sync(0xffffffffu, v.z, step); v.w = __shfl_xor_sync(0xffffffffu, v.w, step);
                            if (up) lo4 = v; else hi4 = v;
                        };
                        swap4(q4[0], q4[1], 1); swap4(q4[2], q4[3], 1);
                        swap4(q4[0], q4[2], 2); swap4(q4[1], q4[3], 2);
                        const int c4 = (lane & 3) * 4, x0 = x - (lane & 3);   // four pixels of a row from x0 on, channels c4 .. c4 + 3
                        float *o1 = o + (long)(y * P.out_w + x0) * P.out_c + n_first[h] + c4;
                        if (y < P.out_h && 16 * h + c4 < n_here)
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                if (x0 + k < P.out_w) *(float4 *)(o1 + (long)k * P.out_c) = q4[k];
                    }
                } else if (inside)   // eight channels of two pixels
#pragma unroll
                    for (int h = 0; h < GC / 16; ++h) {
                        if (16 * h >= n_here) break;
                        float *o2 = o + (long)((y + n_row[h]) * P.out_w + x) * P.out_c + n_first[h];
#pragma unroll
                        for (int p = 0; p < 2; ++p)
#pragma unroll
                            for (int k = 16 * h; k < 16 * h + 16; k += 8)
                                *(float4 *)(o2 + p * P.out_c + (k - 16 * h) / 2) = make_float4(sum[k + p] * scale, sum[k + 2 + p] * scale, sum[k + 4 + p] * scale, sum[k + 6 + p] * scale);
                    }
                continue;
            }
            float *o = P.out + (long)row * P.ldo + y * P.out_w + x;
            if (inside) {
                if (P.pair) {
#pragma unroll
                    for (int j = 0; j < GC; j += 2)
                        if (j < n_here) *(float2 *)(o + col_off[col0 + j]) = make_float2(sum[j] * scale, sum[j + 1] * scale);
                } else {
#pragma unroll
                    for (int j = 0; j < GC; ++j)
                        if (j < n_here && (P.exact || (y + (col_off[NB + col0 + j] >> 4) < P.out_h && x + (col_off[NB + col0 + j] & 15) < P.out_w)))
                            o[col_off[col0 + j]] = sum[j] * scale;
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
}

// ---------------------------------------------------------------- operands
// Largest magnitude of every row (float bits; the caller clears row_max).
__global__ void __launch_bounds__(256) k_row_absmax(int n, const float *__restrict__ A, long lda, unsigned *__restrict__ row_max) {
    pdl_trigger();
    pdl_wait();
    const float *row = A + (long)blockIdx.x * lda;
    float m = 0.f;
    const int j0 = blockIdx.y * 4096, j1 = min(n, j0 + 4096);
    if (((n | lda) & 3) == 0 && ((reinterpret_cast<uintptr_t>(A) & 15) == 0)) {
        for (int j = j0 + threadIdx.x * 4; j < j1; j += 1024) {
            const float4 v = *(const float4 *)(row + j);
            m = fmaxf(fmaxf(fmaxf(m, fabsf(v.x)), fmaxf(fabsf(v.y), fabsf(v.z))), fabsf(v.w));
        }
    } else
        for (int j = j0 + threadIdx.x; j < j1; j += 256) m = fmaxf(m, fabsf(row[j]));
    for (int s = 16; s > 0; s >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
    if ((threadIdx.x & 31) == 0 && m > 0.f) atomicMax(row_max + blockIdx.x, __float_as_uint(m));
}

// Power of two that brings a magnitude into [2^14, 2^15), and its inverse; 1 for zero, infinity and NaN.
__device__ __forceinline__ void win_scale(unsigned bits, float &s, float &inv) {
    const int e = (int)(bits >> 23);   // biased exponent of the magnitude
    if (e == 0 || e == 255) { s = inv = 1.f; return; }
    const int k = 14 - (e - 127);
    // 2^k may leave fp32's range for the smallest magnitudes: clamped (the operand then uses fewer of fp16's binades)
    const int kc = min(max(k, -126), 126);
    s = __uint_as_float((unsigned)(kc + 127) << 23);
    inv = __uint_as_float((unsigned)(127 - kc) << 23);
}

// fp32 rows [C][plane] (channel planes) -> fp16 high and low parts [row][pixel][Cp], scaled by the row's power of two; up
// to 32 channels a pixel's low parts follow its high ones in `hi`.
// 32 pixels x all channels per block.  rpen (optional): the exponent-range share of the contraction's rounding, charged to
// the row: (2^-48 row_max + 1e-37) * q_sum[row / R].  On the way (optional): `bias` added and negative values cut off, the
// result kept in `keep` (it may be A), or values dropped where `mask` is not positive; row_max then holds the rows' largest
// magnitudes before that, and more_max what the bias can add.
struct SplitArgs {
    int C, plane, Cp, R, keep_ld, mask_ld;
    const float *A;
    long lda;
    const unsigned *row_max;
    float more_max;
    const float *bias, *mask;
    float *keep;
    __half *hi, *lo;
    float *row_inv;
    double *rpen;
    const float *q_sum;
};
enum { SPLIT_PLAIN = 0, SPLIT_BIAS = 1, SPLIT_MASK = 2 };
// N elements of a row, zero where there is none.  All loads before the first store and without a branch between them: one element
// behind the other, with both cases looked at each time, they were a chain of that many latencies.  300 images of 64 x 32 x 32 55 us,
// so 32; 210 of 64 x 16 x 16 13.6 and 8.4; one thread a pixel 210 of 16 x 8 x 8 12.6 and 4.1.
template <int WITH, int N>
__device__ __forceinline__ void split_values(const SplitArgs &P, int row, const long (&at)[N], const bool (&in)[N], float (&v)[N]) {
    const float *a = P.A + (long)row * P.lda, *m = WITH == SPLIT_MASK ? P.mask + (long)row * P.mask_ld : P.bias;
    float w[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = in[i] ? a[at[i]] : 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i) w[i] = WITH != SPLIT_PLAIN && in[i] ? m[at[i]] : 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if (WITH == SPLIT_BIAS && in[i]) {
            v[i] = fmaxf(v[i] + w[i], 0.f);
            P.keep[(long)row * P.keep_ld + at[i]] = v[i];
        }
        if (WITH == SPLIT_MASK && !(w[i] > 0.f)) v[i] = 0.f;
    }
}
__device__ __forceinline__ void split_row(const SplitArgs &P, int row, bool first, float &s) {
    const float m = __uint_as_float(P.row_max[row]), bound = P.more_max > 0.f ? __fadd_ru(m, P.more_max) : m;
    float inv;
    win_scale(__float_as_uint(bound), s, inv);
    if (first) {
        P.row_inv[row] = inv;
        if (P.rpen) P.rpen[row] += (3.5527137e-15 * (double)bound + 1e-37) * (double)P.q_sum[row / P.R];
    }
}
template <int WITH>
__global__ void __launch_bounds__(256)
k_split_image(const __grid_constant__ SplitArgs P) {
    extern __shared__ unsigned s_w[];   // [2][32][Cp / 2 + 1] channel pairs; the odd pitch keeps a warp's writes apart
    pdl_trigger();
    pdl_wait();
    const int row = blockIdx.x, p0 = blockIdx.y * 32, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, pitch = P.Cp / 2 + 1, C = P.C, plane = P.plane, Cp = P.Cp;
    float s;
    split_row(P, row, blockIdx.y == 0 && threadIdx.x == 0, s);
    const bool in = p0 + lane < plane;
    for (int first = warp; first < Cp / 2; first += 32) {   // four pairs of channels a thread
        long at[8];
        bool has[8];
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int c = 2 * (first + 8 * (i / 2)) + i % 2;
            at[i] = (long)c * plane + p0 + lane;
            has[i] = in && c < C;
        }
        split_values<WITH>(P, row, at, has, v);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int c2 = first + 8 * u;
            if (c2 >= Cp / 2) break;
            const float v0 = v[2 * u] * s, v1 = v[2 * u + 1] * s;
            const __half2 h = __floats2half2_rn(v0, v1);
            const float2 hf = __half22float2(h);
            const __half2 l = __floats2half2_rn((v0 - hf.x) * 2048.f, (v1 - hf.y) * 2048.f);
            s_w[lane * pitch + c2] = *(const unsigned *)&h;
            s_w[(32 + lane) * pitch + c2] = *(const unsigned *)&l;
        }
    }
    __syncthreads();
    const int n_px = min(32, plane - p0), vec = Cp / 8;   // 16-byte groups per pixel
    const long base = ((long)row * plane + p0) * vec;
    for (int i = threadIdx.x; i < n_px * vec; i += 256) {
        const int px = i / vec, g = i - px * vec;
        const unsigned *a = s_w + px * pitch + g * 4, *b = s_w + (32 + px) * pitch + g * 4;
        if (Cp <= 32) {
            uint4 *px4 = (uint4 *)P.hi + 2 * (base + (long)px * vec);
            px4[g] = make_uint4(a[0], a[1], a[2], a[3]);
            px4[vec + g] = make_uint4(b[0], b[1], b[2], b[3]);
        } else {
            ((uint4 *)P.hi)[base + i] = make_uint4(a[0], a[1], a[2], a[3]);
            ((uint4 *)P.lo)[base + i] = make_uint4(b[0], b[1], b[2], b[3]);
        }
    }
}

// The same up to sixteen channels, one thread a pixel: its pairs are 64 bytes, two whole sectors, and need no exchange (1024
// images of 3 x 32 x 32: 54 -> 22 us, 16 x 16 x 16: 17 -> 10, with bias and ReLU 13, with a mask 14).
template <int WITH>
__global__ void __launch_bounds__(256)
k_split_pixels(const __grid_constant__ SplitArgs P) {
    pdl_trigger();
    pdl_wait();
    const int row = blockIdx.x, px = blockIdx.y * blockDim.x + threadIdx.x;
    float s;
    split_row(P, row, px == 0, s);
    if (px >= P.plane) return;
    unsigned h[8], l[8];
    long from[16];
    bool has[16];
    float v[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) { from[c] = (long)c * P.plane + px; has[c] = c < P.C; }
    split_values<WITH>(P, row, from, has, v);
#pragma unroll
    for (int c2 = 0; c2 < 8; ++c2) {
        const float v0 = v[2 * c2] * s, v1 = v[2 * c2 + 1] * s;
        const __half2 hh = __floats2half2_rn(v0, v1);
        const float2 hf = __half22float2(hh);
        const __half2 ll = __floats2half2_rn((v0 - hf.x) * 2048.f, (v1 - hf.y) * 2048.f);
        h[c2] = *(const unsigned *)&hh; l[c2] = *(const unsigned *)&ll;
    }
    uint4 *at = (uint4 *)P.hi + ((long)row * P.plane + px) * 4;
    at[0] = make_uint4(h[0], h[1], h[2], h[3]); at[1] = make_uint4(h[4], h[5], h[6], h[7]);
    at[2] = make_uint4(l[0], l[1], l[2], l[3]); at[3] = make_uint4(l[4], l[5], l[6], l[7]);
}

// Weights of a window operand: [part][tap][n_blocks * Nb][Cp] fp16, high parts then low parts, zero padded.  sel: how a
// (tap, channel c, column n) maps to W_col [oc x ic*kh*kw]: 0 transposed (c = oc, n = input channel and stride parity), 1 forward (c = ic, n = oc).
// tap_index: tap -> ky*kw+kx; for sel 0 per parity (py, px), -1 where the tap does not reach it.
__global__ void k_win_weights(const float *__restrict__ W, int oc, int ic, int kk, int taps, const int *__restrict__ tap_index, int sel, int st, int NN,
                              int Cp, float scale, __half *__restrict__ out) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x, n_el = (long)taps * NN * Cp;
    if (t >= n_el) return;
    const int c = (int)(t % Cp), n = (int)((t / Cp) % NN), tap = (int)(t / ((long)Cp * NN));
    float w = 0.f;
    const int k = sel == 0 ? 0 : tap_index[tap];
    if (sel == 0) {   // column = (row parity, channel, column parity); a tap serves a parity or it does not
        const int px = n % st, ci = (n / st) % ic, py = n / (st * ic);
        const int kt = py < st ? tap_index[(py * st + px) * taps + tap] : -1;
        if (c < oc && kt >= 0) w = W[((long)c * ic + ci) * kk + kt];
    } else if (c < ic && n < oc) w = W[((long)n * ic + c) * kk + k];
    w *= scale;
    const __half h = __float2half_rn(w);
    out[t] = h;
    out[n_el + t] = __float2half_rn((w - __half2float(h)) * 2048.f);
}

// q_sum[d] = sum of a domain's charge weights over one layer, rounded upwards; one block per domain.
__global__ void __launch_bounds__(256) k_sum_weights(int n, const float *__restrict__ q, long stride, float *__restrict__ q_sum) {
    __shared__ float part[8];
    const float *row = q + (long)blockIdx.x * stride;
    float s = 0.f;
    for (int j = threadIdx.x; j < n; j += 256) s = __fadd_ru(s, row[j]);
    for (int o = 16; o > 0; o >>= 1) s = __fadd_ru(s, __shfl_xor_sync(0xffffffffu, s, o));
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) s = __fadd_ru(s, part[w]);
        q_sum[blockIdx.x] = s;
    }
}

typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                             const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeFn encoder() {
    static EncodeFn fn = nullptr;
    if (fn) return fn;
    void *p = nullptr;
    cudaDriverEntryPointQueryResult qr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) != cudaSuccess || !p) return nullptr;
    return fn = (EncodeFn)p;
}

static CUtensorMapSwizzle swizzle_of(int sw) {
    return sw == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : sw == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
}

double win_eps(const WinOp &op) {
    const Params &P = *(const Params *)op.params;
    const double u23 = 1.1920928955078125e-07, u24 = 5.9604644775390625e-08;
    const int steps = P.taps * P.nchunk * (P.sw / 32);
    const double main_chain = (double)(P.tpc * (P.sw / 32)) * u23;
    const double cross = 2.0 * steps * u23 * 9.765625e-04;   // cross terms are of size 2^-10 S
    const double adds = (double)(P.chains + 1) * u24;       // one addition per chain and the closing one
    return (0.75 * 9.5367431640625e-07 + main_chain + cross + adds) * 1.000001;
}

// Window form of a convolution layer (kind: the `sel` of k_win_weights).  Leaves out->ok false where it does not apply:
// strides over 4, weights that do not fit in shared memory next to three halo tiles, and transposed convolutions whose
// im2col-space product is the faster form.  A tile costs its products whatever part of it lies inside the image, the product
// space what is written there: the line lies at 650 elements of the space per product step of a tile.  A call of 1024
// domains of a classifier of two strided 4x4 convolutions, 8 rows each, us in all; the second one as windows / as products:
//   16 -> 16 channels, side 32 (1820 elements a step) 1130 / 1412   28 (1394) 1288 / 1565   16 (455) 593 / 601
//   32 -> 16           side 32 ( 910)                 1661 / 1875   28 ( 697) 1892 / 2088   16 (228) 742 / 708
//   32 ->  8           side 32 ( 455)                 1610 / 1671   28 ( 348) 1844 / 1866   16 (114) 711 / 622
//   16 ->  8           side 32 ( 910)                 1100 / 1225   28 ( 697) 1242 / 1311   16 (228) 566 / 511
// and the first one (3 input channels): side 32 (683) 1130 / 1333, 28 (523) 1168 / 1285, 16 (341) 601 / 601.  So windows win from
// some 350 elements on; the line stands where products lost to a window kernel of one issuing warp, and shapes from 350 to 650 are
// up to 10 % slower a call than they would be as windows.  Residual blocks lie far on the window's side (64 channels, side 8: 1024 a
// step), and a stem of 64 channels on 3 x 32 x 32 (192) is as fast either way (128 domains of two blocks, 9 rows 10.4 / 10.4 ms).
// The forward form has no such cases.
int win_prepare(nyb200_engine *e, const float *W, float wmax, const ConvGeom &g, int kind, WinOp *out, Carve &c) {
    out->ok = false;
    static_assert(sizeof(Params) <= sizeof(out->params), "parameter storage");
    Params P;
    memset(&P, 0, sizeof(P));
    const int s = g.sh;
    if (g.sh != g.sw || s > 4 || !(wmax > 0.f) || !std::isfinite(wmax)) return NYB200_OK;
    const int Cin = kind == 0 ? g.oc : g.ic;
    P.N = kind == 0 ? g.ic : g.oc;
    P.Cp = Cin <= 16 ? 16 : Cin <= 32 ? 32 : (Cin + 63) / 64 * 64;
    P.sw = std::min(P.Cp, 64) * 2;
    P.swa = P.Cp <= 32 ? P.Cp * 4 : 128;   // high and low parts side by side, or one of them
    P.nchunk = P.Cp > 64 ? P.Cp / 64 : 1;
    P.s = kind == 0 ? s : 1;
    P.in_step = kind == 0 ? 1 : s;
    P.out_c = kind == 0 ? g.ic : P.N;
    P.out_h = kind == 0 ? g.ih : g.oh; P.out_w = kind == 0 ? g.iw : g.ow;
    P.out_plane = P.out_h * P.out_w;
    const int grid_h = (P.out_h + P.s - 1) / P.s, grid_w = (P.out_w + P.s - 1) / P.s;
    P.tiles_y = (grid_h + TY - 1) / TY; P.tiles_x = (grid_w + TX - 1) / TX;
    P.exact = P.out_h % P.s == 0 && P.out_w % P.s == 0;
    std::vector<int> tap_index;   // see k_win_weights
    std::vector<std::pair<int, int>> tap_at;   // halo position of every tap
    int TH = 1, TW = 1;
    if (kind == 0) {
        // One source; the window is the union of the stride parities' windows, every parity a block of columns (a tap a
        // parity does not use has zero weights there: the products of a wider tile cost less than one pass per parity).
        P.N = s * s * g.ic;
        auto span = [&](int k, int pad, int &lo, int &hi) {
            lo = 1 << 30; hi = -(1 << 30);
            for (int p = 0; p < s; ++p) {
                const int k0 = (p + pad) % s, q = (p + pad - k0) / s, n = k0 < k ? (k - k0 + s - 1) / s : 0;
                if (n == 0) continue;   // (pixels that no output reads: a stride larger than the kernel; they come out zero)
                lo = std::min(lo, q - (n - 1)); hi = std::max(hi, q);
            }
        };
        int ylo, yhi, xlo, xhi;
        span(g.kh, g.ph, ylo, yhi); span(g.kw, g.pw, xlo, xhi);
        TH = yhi - ylo + 1; TW = xhi - xlo + 1;
        P.n_src = 1;
        P.src[0].dy = ylo; P.src[0].dx = xlo; P.src[0].ntaps = TH * TW; P.src[0].tap0 = 0; P.src[0].tw = TW;
        for (int h = 0; h < TH; ++h)
            for (int w = 0; w < TW; ++w) tap_at.push_back({h, w});
        for (int py = 0; py < s; ++py)
            for (int px = 0; px < s; ++px)
                for (auto &t : tap_at) {   // oy = yc + ylo + h and oy * s - ph + ky = yc * s + py
                    const int ky = py + g.ph - s * (ylo + t.first), kx = px + g.pw - s * (xlo + t.second);
                    tap_index.push_back(ky >= 0 && ky < g.kh && kx >= 0 && kx < g.kw ? ky * g.kw + kx : -1);
                }
    } else {           // one source per parity of the taps (the input read at the stride)
        for (int ry = 0; ry < s && ry < g.kh; ++ry)
            for (int rx = 0; rx < s && rx < g.kw; ++rx) {
                const int th = (g.kh - ry + s - 1) / s, tw = (g.kw - rx + s - 1) / s;
                Source &so = P.src[P.n_src++];
                so.dy = ry - g.ph; so.dx = rx - g.pw; so.ntaps = th * tw; so.tap0 = (int)tap_at.size(); so.tw = tw;
                for (int h = 0; h < th; ++h)
                    for (int w = 0; w < tw; ++w) { tap_at.push_back({h, w}); tap_index.push_back((ry + s * h) * g.kw + rx + s * w); }
                TH = std::max(TH, th); TW = std::max(TW, tw);
            }
    }
    P.taps = (int)tap_at.size();
    P.bx = TX + TW - 1; P.by = TY + TH - 1;
    if (P.taps > MAXT || P.bx * P.in_step > 256 || P.by * P.in_step > 256) return NYB200_OK;
    const int ksteps = P.sw / 32;
    const long space = (long)g.oh * g.ow * g.ic * g.kh * g.kw, steps = (long)P.taps * P.nchunk * ksteps;
    if (kind == 0 && space < 650 * steps * P.tiles_y * P.tiles_x) return NYB200_OK;
    P.pair = P.s == 2 && P.exact && P.out_w % 2 == 0;
    // pixel-major: a thread's sixteen columns are whole groups of four channels of one pixel, or eight of two
    out->pixel_out = kind == 0 && ((P.s == 1 && P.out_c % 4 == 0) || (P.s == 2 && P.exact && P.out_c % 8 == 0));
    P.slot_bytes = (P.bx * P.by * P.swa + 1023) / 1024 * 1024;
    // columns per CTA: as many as leave room for the weights and three halo buffers
    for (int nb : {64, 32, 16}) {
        if (nb > 16 && nb / 2 >= P.N) continue;
        P.Nb = nb;
        P.n_blocks = (P.N + nb - 1) / nb;
        P.w_tile_bytes = nb * P.sw;
        const long wbytes = (long)P.taps * P.nchunk * 2 * P.w_tile_bytes;
        const long left = (long)SMEM_MOST - 1024 - 1024 - wbytes;
        if (left < 3L * P.slot_bytes) { P.Nb = 0; continue; }
        P.slots = (int)std::min(8L, left / P.slot_bytes);
        break;
    }
    if (P.Nb == 0) return NYB200_OK;
    P.tpc = std::max(1, 4 / ksteps);   // MAIN chains of about four MMA steps
    for (int i = 0; i < P.n_src; ++i) P.chains += P.nchunk * ((P.src[i].ntaps + P.tpc - 1) / P.tpc);
    // weights on the device: parts x taps x columns x channels
    int ex;
    frexpf(wmax, &ex);                       // wmax in [2^(ex-1), 2^ex)
    const float scale = ldexpf(1.f, std::min(15 - ex, 126));
    P.w_inv = 1.f / scale;
    const int NN = P.n_blocks * P.Nb;
    const size_t n_el = (size_t)P.taps * NN * P.Cp;
    out->ok = true;
    void *block = c.take(2 * n_el * 2);
    int *taps_dev = (int *)c.take(tap_index.size() * 4);
    if (!c.block) return NYB200_OK;
    NYB_CUDA(e, cudaMemcpyAsync(taps_dev, tap_index.data(), tap_index.size() * 4, cudaMemcpyHostToDevice, e->stream));   // pageable: staged on return
    k_win_weights<<<(unsigned)((n_el + 255) / 256), 256, 0, e->stream>>>(W, g.oc, g.ic, g.kh * g.kw, P.taps, taps_dev, kind, s, NN, P.Cp, scale,
                                                                        (__half *)block);
    e->launches++;
    EncodeFn enc = encoder();
    if (!enc) return set_err(e, NYB200_ERR_INTERNAL, "cuTensorMapEncodeTiled unavailable");
    cuuint64_t dims[2] = {(cuuint64_t)P.Cp, (cuuint64_t)2 * P.taps * NN}, strides[1] = {(cuuint64_t)P.Cp * 2};
    cuuint32_t box[2] = {(cuuint32_t)std::min(P.Cp, 64), (cuuint32_t)P.Nb}, es[2] = {1, 1};
    if (enc((CUtensorMap *)out->tm_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, block, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
            swizzle_of(P.sw), CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return set_err(e, NYB200_ERR_INTERNAL, "cuTensorMapEncodeTiled failed for a convolution operand");
    out->in_h = kind == 0 ? g.oh : g.ih; out->in_w = kind == 0 ? g.ow : g.iw; out->in_c = Cin; out->in_cp = P.Cp;
    memcpy(out->params, &P, sizeof(P));
    return NYB200_OK;
}

// The window products of `rows` split images hi / lo (scales row_inv) into out [rows x ldo] (channel planes).
int launch_win(nyb200_engine *e, const WinOp &op, int rows, const void *hi, const void *lo, const float *row_inv, float *out, long ldo, int *err,
               bool pixel_major, unsigned *row_max) {
    Params P;
    memcpy(&P, op.params, sizeof(P));
    P.rows = rows; P.row_inv = row_inv; P.out = out; P.ldo = ldo; P.err = err;
    P.pixel_major = pixel_major ? 1 : 0; P.row_max = row_max;
    if (pixel_major && (!op.pixel_out || (ldo & 3) || (reinterpret_cast<uintptr_t>(out) & 15)))
        return set_err(e, NYB200_ERR_INTERNAL, "a convolution's result cannot be pixel-major");
    EncodeFn enc = encoder();
    alignas(64) CUtensorMap tm[2];
    const bool packed = P.Cp <= 32;
    const int row_el = packed ? 2 * P.Cp : P.Cp;   // fp16 values of a pixel in one operand array
    const cuuint64_t dims[4] = {(cuuint64_t)row_el, (cuuint64_t)op.in_w, (cuuint64_t)op.in_h, (cuuint64_t)rows};
    const cuuint64_t strides[3] = {(cuuint64_t)row_el * 2, (cuuint64_t)op.in_w * row_el * 2, (cuuint64_t)op.in_h * op.in_w * row_el * 2};
    const cuuint32_t box[4] = {(cuuint32_t)std::min(row_el, 64), (cuuint32_t)(P.bx * P.in_step), (cuuint32_t)(P.by * P.in_step), 1};
    const cuuint32_t es[4] = {1, (cuuint32_t)P.in_step, (cuuint32_t)P.in_step, 1};
    for (int i = 0; i < 2; ++i)
        if (enc(&tm[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void *>(i && !packed ? lo : hi), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                swizzle_of(P.swa), CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return set_err(e, NYB200_ERR_INTERNAL, "cuTensorMapEncodeTiled failed for an image operand");
    const int sms = usable_sms(e);
    const long tiles = (long)rows * P.tiles_y * P.tiles_x;
    if (tiles > 0x7fffffffL - 65536) return set_err(e, NYB200_ERR_UNSUPPORTED, "batch too large for one convolution");
    const int per_block = (int)std::min<long>(tiles, std::max(1, sms / P.n_blocks));
    if (P.pair && ((ldo & 1) || (reinterpret_cast<uintptr_t>(out) & 7))) P.pair = 0;
    const size_t smem = 1024 + 1024 + (size_t)P.taps * P.nchunk * 2 * P.w_tile_bytes + (size_t)P.slots * P.slot_bytes;
    const dim3 grid((unsigned)(per_block * P.n_blocks));
#define NYB_WIN(KS, NB)                                                                                                     \
    if (P.sw == KS * 32 && P.Nb == NB) {                                                                                    \
        NYB_CUDA(e, cudaFuncSetAttribute(k_conv_win<KS, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MOST));      \
        NYB_CUDA(e, launch_pdl(k_conv_win<KS, NB>, grid, dim3(win::THREADS), smem, e, tm[0], tm[1], *(const CUtensorMap *)op.tm_w, P)); \
    }
    NYB_WIN(1, 16) NYB_WIN(1, 32) NYB_WIN(1, 64) NYB_WIN(2, 16) NYB_WIN(2, 32) NYB_WIN(2, 64) NYB_WIN(4, 16) NYB_WIN(4, 32) NYB_WIN(4, 64)
#undef NYB_WIN
    e->launches++;
    return NYB200_OK;
}

// The operand's place in the workspace, with the words that go with it: row_inv read by the products, row_max written by them.
int win_operand(nyb200_engine *e, const WinOp &op, int rows, void **hi, void **lo, float **row_inv, unsigned **row_max) {
    const size_t n = (size_t)rows * op.in_h * op.in_w * op.in_cp;
    NYB_WS(buf, char *, e, "win_operand", n * 4 + 512);
    NYB_WS(words, unsigned *, e, "win_rows", (size_t)rows * 8);
    *hi = buf;
    *lo = (__half *)buf + ((n + 127) & ~(size_t)127);
    *row_max = words;
    *row_inv = (float *)(words + rows);
    return NYB200_OK;
}

int row_maxima(nyb200_engine *e, int rows, int n, const float *A, long lda, unsigned *row_max) {
    NYB_CUDA(e, cudaMemsetAsync(row_max, 0, (size_t)rows * 4, e->stream));
    NYB_CUDA(e, launch_pdl(k_row_absmax, dim3((unsigned)rows, (unsigned)((n + 4095) / 4096)), dim3(256), 0, e, n, A, lda, row_max));
    e->launches++;
    return NYB200_OK;
}

// A whole convolution of fp32 rows A [rows x lda] (channel planes) into out [rows x ldo]: row magnitudes, split, window
// products.  rpen / q_sum / R: see k_split_image (null where nothing is certified).  with: what happens to the rows on the way.
int conv_win(nyb200_engine *e, const WinOp &op, int rows, const float *A, long lda, float *out, long ldo, double *rpen, const float *q_sum, int R, int *err,
             bool pixel_major, bool report, const WinWith *with) {
    const int plane = op.in_h * op.in_w;
    void *hi, *lo;
    float *row_inv;
    unsigned *row_max;
    NYB_TRY(win_operand(e, op, rows, &hi, &lo, &row_inv, &row_max));
    if (!with || !with->has_max) NYB_TRY(row_maxima(e, rows, op.in_c * plane, A, lda, row_max));
    SplitArgs a;
    memset(&a, 0, sizeof(a));
    a.C = op.in_c; a.plane = plane; a.Cp = op.in_cp; a.R = R; a.A = A; a.lda = lda; a.row_max = row_max;
    a.hi = (__half *)hi; a.lo = (__half *)lo; a.row_inv = row_inv; a.rpen = rpen; a.q_sum = q_sum;
    if (with) {
        a.bias = with->bias; a.keep = with->keep; a.keep_ld = (int)with->keep_ld; a.more_max = with->bias ? with->bias_max : 0.f;
        a.mask = with->mask; a.mask_ld = (int)with->mask_ld;
    }
    const bool by_pixel = op.in_cp == 16;
    const unsigned threads = by_pixel ? (unsigned)std::min(256, (plane + 31) / 32 * 32) : 256;   // (a small image's block is its size)
    const dim3 grid((unsigned)rows, by_pixel ? (plane + threads - 1) / threads : (unsigned)((plane + 31) / 32));
    const size_t smem = by_pixel ? 0 : (size_t)64 * (op.in_cp / 2 + 1) * 4;
    auto split = [&](auto pixels, auto image) { return launch_pdl(by_pixel ? pixels : image, grid, dim3(threads), smem, e, a); };
    if (a.bias && a.mask) return set_err(e, NYB200_ERR_INTERNAL, "a split with a bias and a mask");
    NYB_CUDA(e, a.bias ? split(k_split_pixels<SPLIT_BIAS>, k_split_image<SPLIT_BIAS>) : a.mask ? split(k_split_pixels<SPLIT_MASK>, k_split_image<SPLIT_MASK>)
                                                                                       : split(k_split_pixels<SPLIT_PLAIN>, k_split_image<SPLIT_PLAIN>));
    e->launches++;
    if (report) NYB_CUDA(e, cudaMemsetAsync(row_max, 0, (size_t)rows * 4, e->stream));
    return launch_win(e, op, rows, hi, lo, row_inv, out, ldo, err, pixel_major, report ? row_max : nullptr);
}

int launch_sum_weights(nyb200_engine *e, int D, int n, const float *q, long stride, float *q_sum) {
    k_sum_weights<<<(unsigned)D, 256, 0, e->stream>>>(n, q, stride, q_sum);
    e->launches++;
    return NYB200_OK;
}

}  // namespace nyb
