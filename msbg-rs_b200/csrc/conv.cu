// conv.cu -- block-sparse 3x3x3 convolutions on tcgen05 (see conv.cuh).
#include <algorithm>
#include <type_traits>

#include "conv.cuh"
#include "tc.cuh"

namespace msbg {

constexpr int kConvStages = 3;
constexpr int kWgCells = 64;  // cells (K) per weight-gradient stage

__device__ __forceinline__ uint16_t bf16_rne(float v) { return ElemBF16::store(v); }

// Source row of cell `cell` shifted by tap t, or null when it falls outside
// the active blocks (zero padding).
template <int C>
__device__ __forceinline__ const uint4* tap_row(const ConvLevel& L, const uint16_t* __restrict__ x, int64_t cell, int t) {
    const int lg = L.lg, m = (1 << lg) - 1;
    const int64_t k = cell >> (3 * lg);
    const int v = (int)(cell & ((1 << (3 * lg)) - 1));
    const int gx = (v & m) + t % 3 - 1, gy = ((v >> lg) & m) + (t / 3) % 3 - 1, gz = (v >> (2 * lg)) + t / 9 - 1;
    const int ox = gx < 0 ? 0 : (gx > m ? 2 : 1), oy = gy < 0 ? 0 : (gy > m ? 2 : 1), oz = gz < 0 ? 0 : (gz > m ? 2 : 1);
    const int code = ox + 3 * oy + 9 * oz;
    const int32_t kk = code == 13 ? (int32_t)k : L.nbr27[k * 27 + code];
    if (kk < 0 || kk >= L.n_blocks) return nullptr;  // absent (or a corrupt table entry: read as zero)
    const int64_t c2 = ((int64_t)kk << (3 * lg)) + ((gx & m) | ((gy & m) << lg) | ((gz & m) << (2 * lg)));
    return reinterpret_cast<const uint4*>(x + c2 * C);
}

// Stages of the forward pipeline: four while they fit in 64 KB, else three.
template <int CIN, int COUT>
constexpr int fwd_stages() { return 4 * (128 * CIN * 2 + COUT * CIN * 2) <= 65536 ? 4 : 3; }

template <int CIN, int COUT>
struct FwdSmem {
    static constexpr int STAGES = fwd_stages<CIN, COUT>();
    static constexpr int A_BYTES = 128 * CIN * 2;
    static constexpr int B_BYTES = COUT * CIN * 2;
    static constexpr int OFF_B = STAGES * A_BYTES;
    static constexpr int OFF_BAR = OFF_B + STAGES * B_BYTES;
    static constexpr int BYTES = OFF_BAR + 64;
    // At least 32 KB per CTA: at most 7 CTAs share an SM, so their TMEM
    // columns (<= 64 each) never exceed the 512 an SM has.
    static constexpr int ALLOC = BYTES < 32768 ? 32768 : BYTES;
};

// 16-byte asynchronous copy global -> shared; `present` false writes zeros
// (source size 0: nothing is read from `src`).
__device__ __forceinline__ void cp16_zfill(void* dst, const void* src, bool present) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_u32(dst)), "l"(src),
                 "r"(present ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Epilogue of one output cell: 16 accumulator columns c0 .. c0 + 15, plus
// bias, ReLU, the optional ReLU-derivative mask; bf16 or f32 rows.
template <int COUT>
__device__ __forceinline__ void store16(float* acc, int64_t cell, int c0, const float* __restrict__ bias, int relu,
                                        const uint16_t* __restrict__ mask, int out_f32, int out_ch,
                                        void* __restrict__ y) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        float v = acc[i] + (bias ? __ldg(bias + c0 + i) : 0.0f);
        acc[i] = relu ? fmaxf(v, 0.0f) : v;
    }
    if (mask) {  // ReLU backward: zero where the layer's stored activation is not positive
        const uint4* mk = reinterpret_cast<const uint4*>(mask + cell * COUT + c0);
        uint32_t mw[8];
        *reinterpret_cast<uint4*>(mw) = __ldg(mk);
        *reinterpret_cast<uint4*>(mw + 4) = __ldg(mk + 1);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const uint32_t h = (mw[i >> 1] >> (16 * (i & 1))) & 0xFFFFu;
            if (!(h != 0u && !(h & 0x8000u))) acc[i] = 0.0f;  // bf16 > 0: nonzero, sign clear
        }
    }
    if (out_f32 && out_ch < COUT) {
        float* yo = static_cast<float*>(y) + cell * out_ch + c0;
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (c0 + i < out_ch) yo[i] = acc[i];
    } else if (out_f32) {
        float4* yo = reinterpret_cast<float4*>(static_cast<float*>(y) + cell * COUT + c0);
#pragma unroll
        for (int i = 0; i < 4; ++i) yo[i] = make_float4(acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]);
    } else {
        uint32_t pk[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) pk[i] = (uint32_t)bf16_rne(acc[2 * i]) | ((uint32_t)bf16_rne(acc[2 * i + 1]) << 16);
        uint4* yo = reinterpret_cast<uint4*>(static_cast<uint16_t*>(y) + cell * COUT + c0);
        yo[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        yo[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
    }
}

// Taps flow through STAGES shared-memory stages: the copies of taps t + 1 ..
// t + STAGES - 2 are in flight (cp.async, zero-filled outside the active
// blocks) while the MMAs of tap t run, and a stage is refilled once the MMAs
// that read it (two taps back) have arrived on its mbarrier.
template <int CIN, int COUT>
__global__ void __launch_bounds__(128) conv3_fwd_kernel(ConvLevel L, const uint16_t* __restrict__ x,
                                                        const uint16_t* __restrict__ w, const float* __restrict__ bias,
                                                        int relu, const uint16_t* __restrict__ mask, int out_f32,
                                                        int out_ch, void* __restrict__ y, int* __restrict__ status) {
    using S = FwdSmem<CIN, COUT>;
    constexpr int ST = S::STAGES;
    constexpr int TCOLS = COUT < 32 ? 32 : COUT;
    constexpr int KCH = CIN / 8;
    constexpr uint32_t SBO = KCH * 128;
    constexpr uint32_t IDESC = tc::idesc_bf16(128, COUT, 0, 0);
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::OFF_BAR);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + ST);
    const int tid = threadIdx.x, warp = tid >> 5;
    if (warp == 0) tc::tmem_alloc(tslot, TCOLS);
    if (tid == 0) {
        for (int s = 0; s < ST; ++s) tc::mbar_init(&bars[s], 1);
        tc::fence_mbar_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tslot;

    const int64_t cell = (int64_t)blockIdx.x * 128 + tid;
    const bool valid = cell < L.cells();
    auto issue = [&](int t) {
        const int s = t % ST;
        const uint4* src = valid ? tap_row<CIN>(L, x, cell, t) : nullptr;
        const uint4* from = src ? src : reinterpret_cast<const uint4*>(x);
        uint8_t* arow = smem + s * S::A_BYTES + (tid >> 3) * SBO + (tid & 7) * 16;
#pragma unroll
        for (int j = 0; j < KCH; ++j) cp16_zfill(arow + j * 128, src ? from + j : from, src != nullptr);
        uint8_t* bst = smem + S::OFF_B + s * S::B_BYTES;
        const uint4* wt = reinterpret_cast<const uint4*>(w + (int64_t)t * COUT * CIN);
#pragma unroll
        for (int q = tid; q < COUT * KCH; q += 128) {
            const int n = q / KCH, j = q % KCH;
            cp16_zfill(bst + (n >> 3) * SBO + j * 128 + (n & 7) * 16, wt + q, true);
        }
    };
    constexpr int D = ST - 2;  // prefetch distance in taps
    bool ok = true;
#pragma unroll 1
    for (int t = 0; t < D; ++t) {
        issue(t);
        cp_commit();
    }
#pragma unroll 1
    for (int t = 0; t < 27; ++t) {
        const int s = t % ST;
        cp_wait<D - 1>();  // this thread's copies of tap t have landed
        tc::fence_async_smem();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after_sync();
            const uint32_t a0 = tc::smem_u32(smem + s * S::A_BYTES), b0 = tc::smem_u32(smem + S::OFF_B + s * S::B_BYTES);
#pragma unroll
            for (int kk = 0; kk < CIN / 16; ++kk)
                tc::mma_bf16(tmem, tc::sdesc(a0 + kk * 256, 128, SBO), tc::sdesc(b0 + kk * 256, 128, SBO), IDESC,
                             (t | kk) != 0);
            tc::mma_commit(&bars[s]);
        }
        const int tn = t + D;  // refills the stage of tap tn - ST = t - 2
        if (tn < 27) {
            if (tn >= ST) ok &= tc::mbar_wait(&bars[tn % ST], ((tn - ST) / ST) & 1);
            issue(tn);
        }
        cp_commit();
    }
    ok &= tc::mbar_wait(&bars[26 % ST], (26 / ST) & 1);
    tc::fence_after_sync();
    float acc[16];
#pragma unroll
    for (int c0 = 0; c0 < COUT; c0 += 16) {
        tc::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, acc);
        if (valid && c0 < out_ch) store16<COUT>(acc, cell, c0, bias, relu, mask, out_f32, out_ch, y);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, TCOLS);
    if (!ok && tid == 0) atomicOr(status, 1);
}

// 8^3 blocks (lg = 3), Cin and Cout <= 32: persistent CTAs, one per SM,
// over the blocks.  The weights of all 27 taps are copied into shared memory
// once; per block, its input halo (10^3 rows, each 8-channel chunk of it a
// slab of 16-byte rows in x | y | z order) is copied into one of two halo
// buffers.  Each tap's operand for one z-plane of the block is then a view of
// the halo: 8 groups (y) of 8 rows (x), the groups 160 bytes apart, so one
// lane of warp z issues every MMA of plane z (M = the 64 cells of the plane,
// N = Cout, K = Cin per tap) back to back with no per-tap staging.  Plane z
// of a block accumulates in TMEM columns z * Cout .. of one of two
// accumulators, in the M = 64 data-path layout (row m of the plane in lane
// (m % 16) + 32 (m / 16)).
// While the tensor core works on block i, the threads copy the halo of block
// i + 1 and write out block i - 1.
constexpr int kB8Threads = 512;

template <int CIN, int COUT>
struct B8Smem {
    static constexpr int KCH = CIN / 8;
    static constexpr int SLAB = 1000 * 16;  // one 8-channel chunk of a halo
    static constexpr int HALO = KCH * SLAB;
    static constexpr int B_BYTES = COUT * CIN * 2;
    static constexpr int OFF_W = 2 * HALO;
    static constexpr int OFF_BAR = OFF_W + 27 * B_BYTES;
    static constexpr int BYTES = OFF_BAR + 64;
    static constexpr int ACC_COLS = 8 * COUT;
    static constexpr int TCOLS = 2 * ACC_COLS;
    // More than half of the SM's shared memory: one CTA per SM, so the
    // TMEM columns (up to all 512) are never contended.
    static constexpr int ALLOC = BYTES < 116 * 1024 ? 116 * 1024 : BYTES;
    static constexpr bool FITS = CIN <= 32 && COUT <= 32 && ALLOC <= 227 * 1024;
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(kB8Threads) conv3_b8_kernel(ConvLevel L, const uint16_t* __restrict__ x,
                                                              const uint16_t* __restrict__ w,
                                                              const float* __restrict__ bias, int relu,
                                                              const uint16_t* __restrict__ mask, int out_f32, int out_ch,
                                                              void* __restrict__ y, int* __restrict__ status) {
    using S = B8Smem<CIN, COUT>;
    constexpr int KCH = S::KCH;
    constexpr uint32_t SBO_W = KCH * 128;
    constexpr uint32_t IDESC = tc::idesc_bf16(64, COUT, 0, 0);
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::OFF_BAR);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 2);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // halo of block k into buffer `buf` (zero rows outside the active blocks)
    auto load_halo = [&](int64_t k, int buf) {
        uint8_t* hb = smem + buf * S::HALO;
#pragma unroll 4
        for (int e = tid; e < 1000 * KCH; e += kB8Threads) {
            const int h = e / KCH, j = e % KCH;
            const int gx = h % 10 - 1, gy = (h / 10) % 10 - 1, gz = h / 100 - 1;
            const int ox = gx < 0 ? 0 : (gx > 7 ? 2 : 1), oy = gy < 0 ? 0 : (gy > 7 ? 2 : 1),
                      oz = gz < 0 ? 0 : (gz > 7 ? 2 : 1);
            const int code = ox + 3 * oy + 9 * oz;
            const int32_t kk = code == 13 ? (int32_t)k : __ldg(L.nbr27 + k * 27 + code);
            const bool present = kk >= 0 && kk < L.n_blocks;
            const int64_t c2 = present ? ((int64_t)kk << 9) + ((gx & 7) | ((gy & 7) << 3) | ((gz & 7) << 6)) : 0;
            cp16_zfill(hb + j * S::SLAB + h * 16, reinterpret_cast<const uint4*>(x + c2 * CIN) + j, present);
        }
    };
    for (int e = tid; e < 27 * COUT * KCH; e += kB8Threads) {
        const int t = e / (COUT * KCH), q = e % (COUT * KCH), n = q / KCH, j = q % KCH;
        cp16_zfill(smem + S::OFF_W + t * S::B_BYTES + (n >> 3) * SBO_W + j * 128 + (n & 7) * 16,
                   reinterpret_cast<const uint4*>(w) + e, true);
    }
    const int64_t k0 = blockIdx.x;
    if (k0 < L.n_blocks) load_halo(k0, 0);
    cp_commit();
    if (warp == 0) tc::tmem_alloc(tslot, S::TCOLS);
    if (tid == 0) {
        tc::mbar_init(&bars[0], 8);  // one commit per issuing warp
        tc::mbar_init(&bars[1], 8);
        tc::fence_mbar_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tslot;

    // warps 4g .. 4g + 3 write planes 2g and 2g + 1; lanes 0-15 of warp w
    // hold rows 16 (w % 4) + lane of a plane
    auto epilogue = [&](int64_t k, int buf) {
        __syncwarp();  // tcgen05.ld is warp-wide
        const int m = 16 * (warp & 3) + (lane & 15);
        float acc[16];
#pragma unroll 1
        for (int zz = 0; zz < 2; ++zz) {
            const int z = 2 * (warp >> 2) + zz;
            const int64_t cell = (k << 9) + ((m & 7) | ((m >> 3) << 3) | (z << 6));
#pragma unroll
            for (int c0 = 0; c0 < COUT; c0 += 16) {
                tc::tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(buf * S::ACC_COLS + z * COUT + c0),
                              acc);
                if (lane < 16 && c0 < out_ch) store16<COUT>(acc, cell, c0, bias, relu, mask, out_f32, out_ch, y);
            }
        }
    };

    bool ok = true;
    int i = 0;
    int64_t kprev = -1;
#pragma unroll 1
    for (int64_t k = k0; k < L.n_blocks; k += gridDim.x, ++i) {
        const int buf = i & 1;
        cp_wait<0>();  // this thread's copies of block k's halo (and the weights) have landed
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
        if (lane == 0 && warp < 8) {
            // warp w issues the MMAs of plane w (every offset below is a
            // compile-time constant added to the descriptors' address field)
            const int z = warp;
            const uint64_t a0 = tc::sdesc(tc::smem_u32(smem + buf * S::HALO) + (uint32_t)(z * 1600), S::SLAB, 160);
            const uint64_t b0 = tc::sdesc(tc::smem_u32(smem + S::OFF_W), 128, SBO_W);
            const uint32_t d = tmem + (uint32_t)(buf * S::ACC_COLS + z * COUT);
#pragma unroll 1
            for (int dz = 0; dz < 3; ++dz) {
                // dz * 100: one halo plane (1600 bytes) in the 16-byte units of the address field
                const uint64_t az = a0 + (uint64_t)(dz * 100), bz = b0 + (uint64_t)((dz * 9 * S::B_BYTES) >> 4);
#pragma unroll
                for (int r = 0; r < 9; ++r) {
#pragma unroll
                    for (int kk = 0; kk < CIN / 16; ++kk) {
                        const uint32_t ao = ((r / 3) * 10 + r % 3) * 16 + 2 * kk * S::SLAB;
                        const uint32_t bo = r * S::B_BYTES + kk * 256;
                        tc::mma_bf16(d, az + (ao >> 4), bz + (bo >> 4), IDESC, (dz | r | kk) != 0);
                    }
                }
            }
            tc::mma_commit(&bars[buf]);
        }
        if (kprev >= 0) {
            // block kprev's MMAs (the previous use of the other halo buffer) are done
            ok &= tc::mbar_wait(&bars[buf ^ 1], ((i - 1) >> 1) & 1);
            tc::fence_after_sync();
        }
        if (k + gridDim.x < L.n_blocks) load_halo(k + gridDim.x, buf ^ 1);
        cp_commit();
        if (kprev >= 0) epilogue(kprev, buf ^ 1);
        kprev = k;
    }
    if (kprev >= 0) {
        ok &= tc::mbar_wait(&bars[(i - 1) & 1], ((i - 1) >> 1) & 1);
        tc::fence_after_sync();
        epilogue(kprev, (i - 1) & 1);
    }
    cp_wait<0>();
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, S::TCOLS);
    if (!ok && tid == 0) atomicOr(status, 1);
}

// Copies the input halo of block k, shifted by dx so that its rows are BS
// cells, into shared memory as 16-byte rows of 8 channels: chunk j of the
// cell at halo row (z, y) and column lx goes to
// dst + j * CS + z * ZS + (y * BS + lx) * 16 (zeros outside the active blocks).
// A warp takes a whole row of cells and chunks at a time (or several): the
// row's neighbour blocks come from a lane's register by a shuffle and the
// address is a row base plus a lane constant, about a dozen instructions per
// 32 pieces (worked out per piece they bound the kernels below).  Consecutive
// lanes take pairs of chunks of one cell (a sector); CS is 64 bytes past a
// multiple of 128, so the pairs fall on different banks.
template <int LG, int CIN, int NT, int CS, int ZS>
__device__ __forceinline__ void stage_halo(const ConvLevel& L, const uint16_t* __restrict__ x, int64_t k, int dx, uint8_t* dst) {
    constexpr int BS = 1 << LG, H = BS + 2, NCH = CIN / 8, M = BS - 1;
    constexpr int IPR = BS * NCH;                        // pieces of a row
    constexpr int RPI = IPR < 32 ? 32 / IPR : 1;         // rows a warp takes at once
    constexpr int IPL = IPR > 32 ? IPR / 32 : 1;         // pieces of a row per lane
    static_assert(CS % 128 == 64, "chunk pairs must fall on different banks");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int32_t nb = lane == 13 ? (int32_t)k : lane < 27 ? __ldg(L.nbr27 + k * 27 + lane) : -1;
    const int within = lane % (IPR < 32 ? IPR : 32), sub = lane / (IPR < 32 ? IPR : 32);
#pragma unroll
    for (int h = 0; h < IPL; ++h) {
        const int q = within + 32 * h;
        const int j = (q >> 1) / BS * 2 + (q & 1), lx = (q >> 1) % BS;
        const int gx = lx + dx - 1, ox = gx < 0 ? 0 : (gx >= BS ? 2 : 1);
        const uint16_t* xl = x + (gx & M) * CIN + j * 8;
        uint8_t* dl = dst + j * CS + lx * 16;
#pragma unroll 4
        for (int r0 = warp * RPI; r0 < H * H; r0 += NT / 32 * RPI) {
            const int r = RPI == 1 ? r0 : min(r0 + sub, H * H - 1);  // (a row past the last repeats it)
            const int z = r / H, y = r - z * H;
            const int oy = y == 0 ? 0 : (y == H - 1 ? 2 : 1), oz = z == 0 ? 0 : (z == H - 1 ? 2 : 1);
            const int32_t kk = __shfl_sync(0xffffffffu, nb, ox + 3 * oy + 9 * oz);
            const bool present = kk >= 0 && kk < L.n_blocks;
            const uint32_t cell = ((uint32_t)((y - 1) & M) << LG) | ((uint32_t)((z - 1) & M) << (2 * LG));
            const uint16_t* src = present ? xl + (((int64_t)kk << (3 * LG)) + cell) * CIN : x;
            cp16_zfill(dl + z * ZS + y * (BS * 16), src, present);
        }
    }
}

// 4^3 blocks from staged halos: persistent CTAs, one per SM, over the blocks.
// The work is cut into units (x shift dx, block): the block's input halo
// shifted by dx, so that its rows are BS cells, is copied into one of two
// buffers as 16-byte rows of 8 channels,
//   A [channel chunk][z: BS + 2][y: BS + 2][x: BS].
// The operand of tap (dx, dy, dz) for 128 consecutive rows of the padded plane
// order (z, y of BS + 2, x) is then one contiguous, 16-byte-row view at any
// (dy, dz) shift, so a unit's nine taps need no staging of their own; rows
// with y >= BS (and past the last plane) are computed on whatever lies there
// and ignored.  The nine taps' weights of one dx are in shared memory at a
// time (double-buffered), taken for up to 8 blocks whose accumulators stay in
// TMEM over the three dx.  776 blocks, 64 -> 64 channels (B200): 94 us with
// every tap's rows gathered from global memory, 61 us.  (8^3 blocks run five
// such tiles per block and read shared memory as fast, but copy their halo
// three times: 84 us against 69 us for conv3_b8_kernel, 32 -> 32 channels.)
constexpr int kHaloThreads = 512;

template <int CIN, int COUT>
struct FwdHalo {
    static constexpr int LG = 2, BS = 1 << LG, H = BS + 2, PC = H * BS;
    static constexpr int NCH = CIN / 8, CS = (H * PC * 16) / 128 * 128 + 64 + (H * PC * 16 % 128 > 64 ? 128 : 0);  // bytes of a chunk
    static constexpr int A_BYTES = NCH * CS;
    static constexpr int STAGES = 2;
    static constexpr int W_TAP = COUT * CIN * 2;
    static constexpr int W_BYTES = 2 * 9 * W_TAP;
    static constexpr int GROUP = 8;  // blocks per pass over dx, an accumulator of COUT columns each
    static constexpr int TCOLS = GROUP * COUT;
    static constexpr int OFF_W = STAGES * A_BYTES;
    static constexpr int OFF_BAR = OFF_W + W_BYTES;
    static constexpr int BYTES = OFF_BAR + 64;
    // More than half of the SM's shared memory: one CTA per SM, so the
    // TMEM columns are never contended.
    static constexpr int ALLOC = BYTES < 116 * 1024 ? 116 * 1024 : BYTES;
    static_assert(BS * PC <= 128, "a block's padded cells are the rows of one MMA");
    static_assert(ALLOC <= 227 * 1024 && TCOLS <= 512, "stages or accumulators too large");
    // the last rows of the tile read past their chunk
    static_assert((2 * PC + 2 * BS + 128) * 16 - CS <= W_BYTES, "operand rows past the stages");
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(kHaloThreads) conv3_halo_kernel(ConvLevel L, const uint16_t* __restrict__ x,
                                                                  const uint16_t* __restrict__ w,
                                                                  const float* __restrict__ bias, int relu,
                                                                  const uint16_t* __restrict__ mask, int out_f32, int out_ch,
                                                                  void* __restrict__ y, int* __restrict__ status) {
    using S = FwdHalo<CIN, COUT>;
    constexpr int LG = S::LG, BS = S::BS, H = S::H, PC = S::PC, NCH = S::NCH, ST = S::STAGES;
    constexpr uint32_t SBO_W = NCH * 128;
    constexpr uint32_t IDESC = tc::idesc_bf16(128, COUT, 0, 0);
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::OFF_BAR);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + ST);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // this CTA's blocks k0 .. k0 + nblk - 1, in groups of GROUP; unit u of a
    // group of g blocks is (dx = u / g, block u % g)
    const int64_t k0 = L.n_blocks * blockIdx.x / gridDim.x, k1 = L.n_blocks * (blockIdx.x + 1) / gridDim.x;
    const int nblk = (int)(k1 - k0), units = 3 * nblk;
    if (warp == 0) tc::tmem_alloc(tslot, S::TCOLS);
    if (tid == 0) {
        for (int s = 0; s < ST; ++s) tc::mbar_init(&bars[s], 1);
        tc::fence_mbar_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tslot;

    struct Unit {
        int block, dx, slot;     // block of the CTA, x shift, accumulator
        int pass;                // passes over dx before this one, 3 per group
        bool group_first, group_last;  // first block of its pass, last unit of its group
    };
    auto unit = [&](int u) {
        Unit r;
        const int gi = u / (3 * S::GROUP), v = u - gi * 3 * S::GROUP;
        const int b0 = gi * S::GROUP, g = min(S::GROUP, nblk - b0);
        r.dx = v / g;
        const int b = v - r.dx * g;
        r.block = b0 + b;
        r.slot = b;
        r.pass = 3 * gi + r.dx;
        r.group_first = b == 0;
        r.group_last = v == 3 * g - 1;
        return r;
    };
    auto issue = [&](int u) {
        const Unit r = unit(u);
        const int64_t k = k0 + r.block;
        uint8_t* ast = smem + (u % ST) * S::A_BYTES;
        stage_halo<LG, CIN, kHaloThreads, S::CS, PC * 16>(L, x, k, r.dx, ast);
        // the pass's weights, taps dx + 3 i (the MMAs of the pass before last,
        // whose buffer this is, are done: so are those of unit u - 2)
        if (r.group_first) {
            uint8_t* wst = smem + S::OFF_W + (r.pass & 1) * 9 * S::W_TAP;
            for (int e = tid; e < 9 * COUT * NCH; e += kHaloThreads) {
                const int t = e / (COUT * NCH), q = e % (COUT * NCH), o = q / NCH, j = q % NCH;
                cp16_zfill(wst + t * S::W_TAP + (o >> 3) * SBO_W + j * 128 + (o & 7) * 16,
                           reinterpret_cast<const uint4*>(w) + (int64_t)(r.dx + 3 * t) * (COUT * NCH) + q, true);
            }
        }
    };
    // row m of the tile is padded cell m; four warps write a block
    auto epilogue = [&](int block, int slot) {
        __syncwarp();  // tcgen05.ld is warp-wide
        float acc[16];
        const int q = (warp & 3) * 32 + lane;
        const int cx = q % BS, cy = (q / BS) % H, cz = q / PC;
        const bool valid = cy < BS && cz < BS;
        const int64_t cell = ((k0 + block) << (3 * LG)) + (valid ? cx | (cy << LG) | (cz << (2 * LG)) : 0);
#pragma unroll
        for (int c0 = 0; c0 < COUT; c0 += 16) {
            tc::tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(slot * COUT + c0), acc);
            if (valid && c0 < out_ch) store16<COUT>(acc, cell, c0, bias, relu, mask, out_f32, out_ch, y);
        }
    };
#pragma unroll 1
    for (int u = 0; u < ST - 1; ++u) {
        if (u < units) issue(u);
        cp_commit();
    }
    bool ok = true;
#pragma unroll 1
    for (int u = 0; u < units; ++u) {
        cp_wait<ST - 2>();  // this thread's copies of unit u have landed
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        const Unit r = unit(u);
        if (tid == 0) {
            tc::fence_after_sync();
            const uint64_t a0 = tc::sdesc(tc::smem_u32(smem + (u % ST) * S::A_BYTES), S::CS, 128);
            const uint64_t b0 = tc::sdesc(tc::smem_u32(smem + S::OFF_W + (r.pass & 1) * 9 * S::W_TAP), 128, SBO_W);
            const uint32_t d = tmem + (uint32_t)(r.slot * COUT);
#pragma unroll 1
            for (int dz = 0; dz < 3; ++dz) {
#pragma unroll
                for (int dy = 0; dy < 3; ++dy) {
#pragma unroll
                    for (int kk = 0; kk < CIN / 16; ++kk) {
                        // offsets in the 16-byte units of the descriptors' address field
                        const uint64_t ao = (uint64_t)(dz * PC + dy * BS) + (uint64_t)((2 * kk * S::CS) >> 4);
                        const uint64_t bo = (uint64_t)(((3 * dz + dy) * S::W_TAP + kk * 256) >> 4);
                        tc::mma_bf16(d, a0 + ao, b0 + bo, IDESC, (r.dx | dz | dy | kk) != 0);
                    }
                }
            }
            tc::mma_commit(&bars[u % ST]);
        }
        // with this unit's MMAs queued, the stage of the unit before (whose
        // MMAs have then read it) is filled again
        const int nxt = u + ST - 1;
        if (nxt < units) {
            if (u >= 1) ok &= tc::mbar_wait(&bars[nxt % ST], ((u - 1) / ST) & 1);
            issue(nxt);
        }
        cp_commit();
        if (r.group_last) {  // the group's blocks, a set of four warps each
            ok &= tc::mbar_wait(&bars[u % ST], (u / ST) & 1);
            tc::fence_after_sync();
            for (int b = warp >> 2; b <= r.slot; b += kHaloThreads / 128) epilogue(r.block - r.slot + b, b);
        }
    }
    cp_wait<0>();
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, S::TCOLS);
    if (!ok && tid == 0) atomicOr(status, 1);
}

template <int CIN, int COUT>
struct WgSmem {
    static constexpr int A_BYTES = 128 * kWgCells * 2;
    static constexpr int B_BYTES = COUT * kWgCells * 2;
    static constexpr int OFF_B = kConvStages * A_BYTES;
    static constexpr int OFF_BAR = OFF_B + kConvStages * B_BYTES;
    static constexpr int BYTES = OFF_BAR + 64;
    static constexpr int ALLOC = BYTES < 32768 ? 32768 : BYTES;
};

// partial[part][q][o], q = tap * CIN + i over tiles of 128 (rows past
// 27 * CIN are zero).
template <int CIN, int COUT>
__global__ void __launch_bounds__(128) conv3_wgrad_kernel(ConvLevel L, const uint16_t* __restrict__ x,
                                                          const uint16_t* __restrict__ dy, int64_t cells_per_part,
                                                          float* __restrict__ partial, int* __restrict__ status) {
    using S = WgSmem<CIN, COUT>;
    constexpr int TCOLS = COUT < 32 ? 32 : COUT;
    constexpr uint32_t SBO = (kWgCells / 8) * 128;
    constexpr uint32_t IDESC = tc::idesc_bf16(128, COUT, 1, 1);
    constexpr int TPT = 128 / CIN;  // taps per M tile
    constexpr int MROWS = ((27 * CIN + 127) / 128) * 128;
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::OFF_BAR);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + kConvStages);
    const int tid = threadIdx.x, warp = tid >> 5;
    if (warp == 0) tc::tmem_alloc(tslot, TCOLS);
    if (tid == 0) {
        for (int s = 0; s < kConvStages; ++s) tc::mbar_init(&bars[s], 1);
        tc::fence_mbar_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tslot;

    const int mt = blockIdx.x, part = blockIdx.y;
    const int tap0 = mt * TPT;
    const int64_t total = L.cells();
    const int64_t c_begin = (int64_t)part * cells_per_part;
    const int64_t c_end = std::min<int64_t>(total, c_begin + cells_per_part);
    const int nchunks = c_end > c_begin ? (int)((c_end - c_begin + kWgCells - 1) / kWgCells) : 0;
    bool ok = true;
    for (int ch = 0; ch < nchunks; ++ch) {
        const int s = ch % kConvStages;
        if (ch >= kConvStages) ok &= tc::mbar_wait(&bars[s], ((ch / kConvStages) - 1) & 1);
        const int64_t cbase = c_begin + (int64_t)ch * kWgCells;
        uint8_t* ast = smem + s * S::A_BYTES;
#pragma unroll 4
        for (int r = 0; r < (kWgCells * 16) / 128; ++r) {
            const int item = tid + 128 * r;
            const int c = item % kWgCells, mg = item / kWgCells;
            const int64_t cell = cbase + c;
            const int q0 = mg * 8;
            const int tap = tap0 + q0 / CIN, ci0 = q0 % CIN;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (cell < c_end && tap < 27) {
                const uint4* src = tap_row<CIN>(L, x, cell, tap);
                if (src) v = __ldg(src + ci0 / 8);
            }
            *reinterpret_cast<uint4*>(ast + mg * SBO + (c >> 3) * 128 + (c & 7) * 16) = v;
        }
        uint8_t* bst = smem + S::OFF_B + s * S::B_BYTES;
        for (int item = tid; item < kWgCells * (COUT / 8); item += 128) {
            const int c = item % kWgCells, ng = item / kWgCells;
            const int64_t cell = cbase + c;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (cell < c_end) v = __ldg(reinterpret_cast<const uint4*>(dy + cell * COUT) + ng);
            *reinterpret_cast<uint4*>(bst + ng * SBO + (c >> 3) * 128 + (c & 7) * 16) = v;
        }
        tc::fence_async_smem();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after_sync();
            const uint32_t a0 = tc::smem_u32(ast), b0 = tc::smem_u32(bst);
#pragma unroll
            for (int kk = 0; kk < kWgCells / 16; ++kk)
                tc::mma_bf16(tmem, tc::sdesc(a0 + kk * 256, 128, SBO), tc::sdesc(b0 + kk * 256, 128, SBO), IDESC,
                             (ch | kk) != 0);
            tc::mma_commit(&bars[s]);
        }
    }
    if (nchunks > 0) {
        ok &= tc::mbar_wait(&bars[(nchunks - 1) % kConvStages], ((nchunks - 1) / kConvStages) & 1);
        tc::fence_after_sync();
    }
    float acc[16];
    const int q = mt * 128 + tid;
    float* out = partial + ((int64_t)part * MROWS + q) * COUT;
#pragma unroll
    for (int c0 = 0; c0 < COUT; c0 += 16) {
        if (nchunks > 0) {
            tc::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, acc);
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[i] = 0.0f;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            reinterpret_cast<float4*>(out + c0)[i] = make_float4(acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, TCOLS);
    if (!ok && tid == 0) atomicOr(status, 1);
}

// Weight gradient on 8^3 and 4^3 blocks from staged halos.  CTA (dx, part)
// forms the nine taps of one x shift over a range of whole blocks: per block
// it copies the input halo, shifted by dx so that its rows are BS cells, and
// the block's output gradient into shared memory once (STAGES blocks in
// flight), as 16-byte rows of 8 channels:
//   A [z: BS + 2][channel chunk][y: BS + 2][x: BS],  B [chunk][cell].
// Sixteen consecutive cells of a plane are then 256 contiguous bytes, one
// K = 16 step, at any y shift; and the chunks of a plane and of the planes
// after it follow at one stride, so one MMA of M = 128 rows takes 128 / CIN
// dz shifts at once (rows beyond dz = 2 are computed on whatever lies there
// and ignored).  Three warps issue the three dy shifts' MMAs, alternating
// between two accumulators each where TMEM has room.
// The kernel it replaces gathered every tap's operand from global memory
// (27 reads of each input row, index arithmetic per 16 bytes, nothing in
// flight over its barrier).  Weight gradient of 776 blocks (B200), 8^3 cells,
// 32 -> 32 channels: 523 -> 79 us; 4^3, 64 -> 64: 191 -> 42 us.
template <int LG, int CIN, int COUT>
struct WgHalo {
    static constexpr int BS = 1 << LG, H = BS + 2, PC = H * BS;  // cells of a staged plane
    static constexpr int NCH = CIN / 8, NCO = COUT / 8, CELLS = BS * BS * BS;
    static constexpr int CS = PC * 16 / 128 * 128 + 64 + (PC * 16 % 128 > 64 ? 128 : 0);  // bytes of a chunk of a plane
    static constexpr int A_BYTES = H * NCH * CS, B_BYTES = NCO * CELLS * 16;
    static constexpr int STAGES = LG == 2 ? 4 : 2;
    static constexpr int OFF_B = STAGES * A_BYTES;
    static constexpr int OFF_BAR = OFF_B + STAGES * B_BYTES;
    static constexpr int BYTES = OFF_BAR + 64;
    static constexpr int PPM = 128 / CIN;            // dz shifts of one MMA
    static constexpr int NM = (3 + PPM - 1) / PPM;   // MMAs for the three
    static constexpr int COLS1 = 3 * NM * COUT;      // accumulator columns of the CTA's taps
    static constexpr int NACC = 2 * COLS1 <= 512 ? 2 : 1;
    static constexpr int TCOLS = NACC * COLS1 <= 128 ? 128 : NACC * COLS1 <= 256 ? 256 : 512;
    // the last M rows of the last planes read past the A stages
    static constexpr int PAST = ((BS - 1 + (NM - 1) * PPM) * NCH + 16) * CS + 2 * BS * 16;
    // More than half of the SM's shared memory: one CTA per SM, so the TMEM
    // columns are never contended.
    static constexpr int ALLOC = BYTES < 116 * 1024 ? 116 * 1024 : BYTES;
    static constexpr bool FITS = ALLOC <= 227 * 1024 && PAST - A_BYTES <= STAGES * B_BYTES && COLS1 <= 512;
};
constexpr int kWgThreads = 512;

template <int LG, int CIN, int COUT>
__global__ void __launch_bounds__(kWgThreads) conv3_wgrad_halo_kernel(ConvLevel L, const uint16_t* __restrict__ x,
                                                                      const uint16_t* __restrict__ dy, float* __restrict__ partial,
                                                                      int* __restrict__ status) {
    using S = WgHalo<LG, CIN, COUT>;
    constexpr int BS = S::BS, NCH = S::NCH, ST = S::STAGES;
    constexpr int MROWS = ((27 * CIN + 127) / 128) * 128;
    constexpr int KSTEPS = S::CELLS / 16, KPP = BS * BS / 16;  // K steps of a block, of a plane
    constexpr uint32_t IDESC = tc::idesc_bf16(128, COUT, 1, 1);
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::OFF_BAR);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + ST);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int dx = blockIdx.x, part = blockIdx.y;
    const int64_t k0 = L.n_blocks * part / gridDim.y, k1 = L.n_blocks * (part + 1) / gridDim.y;
    const int nblk = (int)(k1 - k0);
    if (warp == 0) tc::tmem_alloc(tslot, S::TCOLS);
    if (tid == 0) {
        for (int s = 0; s < ST; ++s) tc::mbar_init(&bars[s], 3);  // one commit per issuing warp
        tc::fence_mbar_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tslot;

    // Block k0 + i into its stage
    auto issue = [&](int i) {
        const int64_t k = k0 + i;
        stage_halo<LG, CIN, kWgThreads, S::CS, NCH * S::CS>(L, x, k, dx, smem + (i % ST) * S::A_BYTES);
        uint8_t* bst = smem + S::OFF_B + (i % ST) * S::B_BYTES;
        const uint4* src = reinterpret_cast<const uint4*>(dy + (k << (3 * LG)) * COUT);
#pragma unroll 4
        for (int e = tid; e < S::NCO * S::CELLS; e += kWgThreads) {
            const int g = (e >> 4) / (S::NCO / 2), j = ((e >> 4) % (S::NCO / 2)) * 2 + (e & 1), c = g * 8 + ((e >> 1) & 7);
            cp16_zfill(bst + (j * S::CELLS + c) * 16, src + c * S::NCO + j, true);
        }
    };
#pragma unroll 1
    for (int i = 0; i < ST - 1; ++i) {
        if (i < nblk) issue(i);
        cp_commit();
    }
    bool ok = true;
#pragma unroll 1
    for (int i = 0; i < nblk; ++i) {
        cp_wait<ST - 2>();  // this thread's copies of block i have landed
        tc::fence_async_smem();
        __syncthreads();
        if (lane == 0 && warp < 3) {
            tc::fence_after_sync();
            const uint32_t a0 = tc::smem_u32(smem + (i % ST) * S::A_BYTES) + (uint32_t)(warp * BS * 16);  // dy = warp
            const uint32_t b0 = tc::smem_u32(smem + S::OFF_B + (i % ST) * S::B_BYTES);
#pragma unroll 4
            for (int kk = 0; kk < KSTEPS; ++kk) {
                const int z = kk / KPP, acc = kk % S::NACC;
                const uint64_t bd = tc::sdesc(b0 + (uint32_t)(kk * 256), 128, S::CELLS * 16);
#pragma unroll
                for (int nm = 0; nm < S::NM; ++nm) {
                    const uint64_t ad = tc::sdesc(a0 + (uint32_t)((z + nm * S::PPM) * NCH * S::CS + (kk % KPP) * 256), 128, S::CS);
                    tc::mma_bf16(tmem + (uint32_t)(((acc * 3 + warp) * S::NM + nm) * COUT), ad, bd, IDESC, i > 0 || kk >= S::NACC);
                }
            }
            tc::mma_commit(&bars[i % ST]);
        }
        // with this block's MMAs queued, the stage of the block before (whose
        // MMAs have then read it) is filled again
        const int nxt = i + ST - 1;
        if (nxt < nblk) {
            if (i >= 1) ok &= tc::mbar_wait(&bars[nxt % ST], ((i - 1) / ST) & 1);
            issue(nxt);
        }
        cp_commit();
    }
    if (nblk > 0) {
        ok &= tc::mbar_wait(&bars[(nblk - 1) % ST], ((nblk - 1) / ST) & 1);
        tc::fence_after_sync();
    }
    if (warp < 4) {
        __syncwarp();  // tcgen05.ld is warp-wide
        const int m = tid;  // row: dz shift m / CIN of its MMA, input channel m % CIN
#pragma unroll 1
        for (int d = 0; d < 3; ++d) {
#pragma unroll 1
            for (int nm = 0; nm < S::NM; ++nm) {
                const int dz = nm * S::PPM + m / CIN;
                float* out = partial + ((int64_t)part * MROWS + (dx + 3 * d + 9 * dz) * CIN + m % CIN) * COUT;
#pragma unroll 1
                for (int c0 = 0; c0 < COUT; c0 += 16) {
                    float v[16];
#pragma unroll
                    for (int q = 0; q < 16; ++q) v[q] = 0.0f;
                    if (nblk > 0) {
                        float t[16];
                        tc::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)((d * S::NM + nm) * COUT + c0), v);
                        if (S::NACC == 2) {
                            tc::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(((3 + d) * S::NM + nm) * COUT + c0), t);
#pragma unroll
                            for (int q = 0; q < 16; ++q) v[q] += t[q];
                        }
                    }
                    if (dz < 3) {
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            reinterpret_cast<float4*>(out + c0)[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                    }
                }
            }
        }
    }
    cp_wait<0>();
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, S::TCOLS);
    if (!ok && tid == 0) atomicOr(status, 1);
}

// dw[t][o][i] (+)= sum over parts (in order) of partial[part][t * CIN + i][o]
__global__ void conv3_wgrad_reduce_kernel(const float* __restrict__ partial, int parts, int cin, int cout, int mrows,
                                          float* __restrict__ dw, int acc) {
    const int n = 27 * cin * cout;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        const int i = e % cin, o = (e / cin) % cout, t = e / (cin * cout);
        const int q = t * cin + i;
        float s = 0.0f;
        for (int p = 0; p < parts; ++p) s += partial[((int64_t)p * mrows + q) * cout + o];
        dw[e] = acc ? dw[e] + s : s;
    }
}

template <int CIN, int COUT>
static void launch_fwd(msbg_ctx* ctx, const ConvLevel& L, const uint16_t* x, const uint16_t* w, const float* bias, bool relu,
                       const uint16_t* mask, bool out_f32, int out_ch, void* y) {
    using S = FwdSmem<CIN, COUT>;
    static bool attr = false;
    if (!attr) {
        CUDA_CHECK(cudaFuncSetAttribute(conv3_fwd_kernel<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::ALLOC));
        attr = true;
    }
    const int64_t cells = L.cells();
    if (!cells) return;
    if constexpr (B8Smem<CIN, COUT>::FITS) {
        if (L.lg == 3) {
            using S8 = B8Smem<CIN, COUT>;
            static bool attr8 = false;
            if (!attr8) {
                CUDA_CHECK(cudaFuncSetAttribute(conv3_b8_kernel<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                S8::ALLOC));
                attr8 = true;
            }
            static int sms = 0;
            if (!sms) CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
            begin_launch(ctx);
            const unsigned grid = (unsigned)std::min<int64_t>(L.n_blocks, sms);
            conv3_b8_kernel<CIN, COUT><<<grid, kB8Threads, S8::ALLOC, ctx->stream>>>(
                L, x, w, bias, relu ? 1 : 0, mask, out_f32 ? 1 : 0, out_ch > 0 ? out_ch : COUT, y, ctx->status.as<int>());
            after_launch(ctx, "conv3_b8_kernel");
            return;
        }
    }
    if (L.lg == 2) {
        using H = FwdHalo<CIN, COUT>;
        static bool hattr = false;
        if (!hattr) {
            CUDA_CHECK(cudaFuncSetAttribute(conv3_halo_kernel<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, H::ALLOC));
            hattr = true;
        }
        static int sms = 0;
        if (!sms) CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
        begin_launch(ctx);
        conv3_halo_kernel<CIN, COUT><<<(unsigned)std::min<int64_t>(L.n_blocks, sms), kHaloThreads, H::ALLOC, ctx->stream>>>(
            L, x, w, bias, relu ? 1 : 0, mask, out_f32 ? 1 : 0, out_ch > 0 ? out_ch : COUT, y, ctx->status.as<int>());
        after_launch(ctx, "conv3_halo_kernel");
        return;
    }
    begin_launch(ctx);
    conv3_fwd_kernel<CIN, COUT><<<(unsigned)((cells + 127) / 128), 128, S::ALLOC, ctx->stream>>>(
        L, x, w, bias, relu ? 1 : 0, mask, out_f32 ? 1 : 0, out_ch > 0 ? out_ch : COUT, y, ctx->status.as<int>());
    after_launch(ctx, "conv3_fwd_kernel");
}

template <int CIN, int COUT>
static void launch_wgrad(msbg_ctx* ctx, const ConvLevel& L, const uint16_t* x, const uint16_t* dy, float* dw, bool acc) {
    using S = WgSmem<CIN, COUT>;
    static bool attr = false;
    if (!attr) {
        CUDA_CHECK(cudaFuncSetAttribute(conv3_wgrad_kernel<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::ALLOC));
        attr = true;
    }
    constexpr int MT = (27 * CIN + 127) / 128;
    constexpr int MROWS = MT * 128;
    const int64_t cells = L.cells();
    // 8^3 and 4^3 blocks whose stages fit shared memory: from staged halos,
    // one CTA per SM over the three x shifts
    auto from_halos = [&](auto lg) {
        constexpr int LG = decltype(lg)::value;
        using W = WgHalo<LG, CIN, COUT>;
        if constexpr (W::FITS) {
            static bool wattr = false;
            if (!wattr) {
                CUDA_CHECK(cudaFuncSetAttribute(conv3_wgrad_halo_kernel<LG, CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                W::ALLOC));
                wattr = true;
            }
            const int parts = (int)std::max<int64_t>(1, std::min<int64_t>(L.n_blocks, 148 / 3));
            ScratchLayout SL;
            const size_t op = SL.add<float>((size_t)parts * MROWS * COUT);
            float* partial = ScratchLayout::at<float>(scratch(ctx, SL), op);
            begin_launch(ctx);
            conv3_wgrad_halo_kernel<LG, CIN, COUT><<<dim3(3, (unsigned)parts), kWgThreads, W::ALLOC, ctx->stream>>>(
                L, x, dy, partial, ctx->status.as<int>());
            after_launch(ctx, "conv3_wgrad_halo_kernel");
            begin_launch(ctx);
            conv3_wgrad_reduce_kernel<<<(27 * CIN * COUT + 255) / 256, 256, 0, ctx->stream>>>(partial, parts, CIN, COUT, MROWS, dw,
                                                                                               acc ? 1 : 0);
            after_launch(ctx, "conv3_wgrad_reduce_kernel");
            return true;
        } else {
            return false;
        }
    };
    // A few blocks leave its few CTAs a block's latency each, and the many small
    // CTAs of the gather kernel finish earlier (a call with its host round trip, B200,
    // gather against halos: 4^3, 64 -> 64 channels, 8 blocks 30.9 / 33.9 us, 20
    // 38.2 / 39.1, 40 54.1 / 47.2; 16 and 32 input channels in halos' favour from one
    // block on; 8^3, 32 -> 32, one block 27.0 / 28.1, three 30.1 / 28.3).
    const bool few = L.lg == 3 ? L.n_blocks < 2 : CIN >= 64 && L.n_blocks < 20;
    if (!few && L.lg == 3 && from_halos(std::integral_constant<int, 3>())) return;
    if (!few && L.lg == 2 && from_halos(std::integral_constant<int, 2>())) return;
    // about 4 CTAs per SM in total, each over a contiguous range of whole 64-cell chunks
    const int64_t chunks = std::max<int64_t>(1, (cells + kWgCells - 1) / kWgCells);
    const int parts = (int)std::min<int64_t>(chunks, std::max<int64_t>(1, 592 / MT));
    const int64_t cells_per_part = ((chunks + parts - 1) / parts) * kWgCells;
    ScratchLayout SL;
    const size_t op = SL.add<float>((size_t)parts * MROWS * COUT);
    float* partial = ScratchLayout::at<float>(scratch(ctx, SL), op);
    begin_launch(ctx);
    conv3_wgrad_kernel<CIN, COUT><<<dim3(MT, parts), 128, S::ALLOC, ctx->stream>>>(L, x, dy, cells_per_part, partial,
                                                                                  ctx->status.as<int>());
    after_launch(ctx, "conv3_wgrad_kernel");
    begin_launch(ctx);
    conv3_wgrad_reduce_kernel<<<(27 * CIN * COUT + 255) / 256, 256, 0, ctx->stream>>>(partial, parts, CIN, COUT, MROWS, dw,
                                                                                       acc ? 1 : 0);
    after_launch(ctx, "conv3_wgrad_reduce_kernel");
}

#define MSBG_CONV_PAIRS(X) X(16, 32) X(32, 16) X(32, 32) X(32, 64) X(64, 32) X(64, 64) X(16, 16) X(64, 16) X(16, 64)

void conv3_forward(msbg_ctx* ctx, const ConvLevel& L, int cin, int cout, const uint16_t* x, const uint16_t* w,
                   const float* bias, bool relu, bool out_f32, void* y, const uint16_t* mask, int out_ch) {
    MSBG_REQUIRE(out_ch >= 0 && out_ch <= cout && (out_f32 || out_ch == 0 || out_ch == cout), "conv3: bad output width");
#define MSBG_FWD_CASE(A, B) \
    if (cin == A && cout == B) return launch_fwd<A, B>(ctx, L, x, w, bias, relu, mask, out_f32, out_ch, y);
    MSBG_CONV_PAIRS(MSBG_FWD_CASE)
#undef MSBG_FWD_CASE
    MSBG_THROW(MSBG_ERR_ARG, "conv3: channel counts must be 16, 32 or 64");
}

void conv3_wgrad(msbg_ctx* ctx, const ConvLevel& L, int cin, int cout, const uint16_t* x, const uint16_t* dy, float* dw,
                 bool acc) {
#define MSBG_WG_CASE(A, B) \
    if (cin == A && cout == B) return launch_wgrad<A, B>(ctx, L, x, dy, dw, acc);
    MSBG_CONV_PAIRS(MSBG_WG_CASE)
#undef MSBG_WG_CASE
    MSBG_THROW(MSBG_ERR_ARG, "conv3: channel counts must be 16, 32 or 64");
}

}  // namespace msbg

using namespace msbg;

extern "C" {

int msbg_conv3_forward_device(msbg_ctx* ctx, const int32_t* d_nbr27, int64_t n_blocks, int lg, int cin, int cout,
                              const uint16_t* d_x, const uint16_t* d_w, const float* d_bias, int relu, int out_f32,
                              void* d_y) {
    MSBG_API_BEGIN
    MSBG_REQUIRE(ctx && d_nbr27 && d_x && d_w && d_y && n_blocks >= 0 && lg >= 1 && lg <= 5, "bad argument");
    set_device(ctx);
    conv3_forward(ctx, ConvLevel{d_nbr27, lg, n_blocks}, cin, cout, d_x, d_w, d_bias, relu != 0, out_f32 != 0, d_y);
    check_device_status(ctx);
    MSBG_API_END
}

int msbg_conv3_wgrad_device(msbg_ctx* ctx, const int32_t* d_nbr27, int64_t n_blocks, int lg, int cin, int cout,
                            const uint16_t* d_x, const uint16_t* d_dy, float* d_dw) {
    MSBG_API_BEGIN
    MSBG_REQUIRE(ctx && d_nbr27 && d_x && d_dy && d_dw && n_blocks >= 0 && lg >= 1 && lg <= 5, "bad argument");
    set_device(ctx);
    conv3_wgrad(ctx, ConvLevel{d_nbr27, lg, n_blocks}, cin, cout, d_x, d_dy, d_dw, false);
    check_device_status(ctx);
    MSBG_API_END
}

}  // extern "C"
