// k_learned.cu -- the learned preconditioner's kernels on sm_100a.
//
// Convolutions are implicit GEMMs on the 5th-generation tensor cores:
//   forward / input gradient: D[voxel][cout] += A[voxel][cin] * B[cout][cin]
//     per tap; M = 128 voxels per CTA, N = cout (16/32/64), K = 27 taps x cin.
//     A rows are gathered (zero padding at the grid edge) from channels-last
//     BF16 activations into shared memory in the UMMA K-major core-matrix
//     layout; B is the tap's pre-formatted weight tile.
//   weight gradient: D[cout][cin] += A[cout][voxel] * B[cin][voxel] per tap
//     with K = voxels; both operands are MN-major, which is what
//     channels-last activations already are, so each voxel's channels are
//     one 16-byte shared-memory store.
// One thread issues tcgen05.mma into a TMEM accumulator; tcgen05.commit
// arrives on an mbarrier; the epilogue reads TMEM with tcgen05.ld.  The
// gathering kernel (k_conv) stages two taps at a time; the brick kernel
// (k_conv_brick, every layer of this network) stages each output tile's
// input brick once by TMA and runs its tiles as a warp-specialised pipeline
// over two accumulators.  The solver's forward passes run tile-sparse: a
// plan (plan_sparse) lists, per stage, the tiles the cells with type != 0
// depend on.
// Every mbarrier wait is bounded: on timeout the kernel records it in
// NetStatus, waits (bounded) for its own copies and MMAs in flight, frees
// TMEM and returns.
#include <algorithm>
#include <cmath>
#include <random>

#include "net.cuh"
#include "lhi.h"
#include "tma.cuh"

namespace lhi {

namespace {

// ------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait for the completion of the barrier phase with this parity:
// non-blocking test_wait polled against a 200 ms deadline.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity) {
    const uint32_t addr = smem_u32(bar);
    const uint64_t deadline = global_ns() + 200000000ull;
    for (;;) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
        if (global_ns() > deadline) return false;
    }
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// warp-wide
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// UMMA shared-memory descriptor, no swizzle (canonical INTERLEAVE layout):
// start address, leading (K-direction) and stride (M/N-direction) byte
// offsets between 8 x 16-byte core matrices, version 1.
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= uint64_t((saddr >> 4) & 0x3FFFu);
    d |= uint64_t((lbo >> 4) & 0x3FFFu) << 16;
    d |= uint64_t((sbo >> 4) & 0x3FFFu) << 32;
    d |= uint64_t(1) << 46;
    return d;
}

// Instruction descriptor of kind::f16: BF16 x BF16 -> F32, M x N.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N, int a_mn, int b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(a_mn) << 15) | (uint32_t(b_mn) << 16) |
           (uint32_t(N >> 3) << 17) | (uint32_t(M >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
    const uint32_t z = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
        :
        : "r"(d_tmem), "l"(ad), "l"(bd), "r"(idesc), "r"(acc), "r"(z), "r"(z), "r"(z), "r"(z)
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// warp-collective: callers reconverge the warp first (__syncwarp)
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = __uint_as_float(r[k]);
}

__device__ __forceinline__ void tap_offset(int tap, int& dx, int& dy, int& dz) {
    dx = tap / 9 - 1;
    dy = (tap / 3) % 3 - 1;
    dz = tap % 3 - 1;
}

// ------------------------------------------------------------ convolution
constexpr int kConvM = 128;  // voxels per CTA

struct ConvParams {
    const uint16_t* in;   // channels-last BF16, cin channels
    int cin;              // padded: 16, 32 or 64
    const uint16_t* w;    // 27 formatted B tiles [cout][cin]
    int cout;             // padded: 16, 32 or 64
    const float* bias;    // cout_real entries or null
    int cout_real;
    int nx, ny, nz;
    long long nvox;
    int mode;             // 0: BF16 out (+bias +skip, relu); 1: FP32 out, all channels; 2: FP32 channel 0 + bias
    const uint16_t* skip; // BF16, cout channels (mode 0), or null
    int relu;
    uint16_t* out_b;
    float* out_f;
    NetStatus* status;
    const int32_t* tiles;  // brick kernel: the output tiles to evaluate (indices as the dense loop's), or null: all
    const int* ntiles;     // their count (device)
};

// Epilogue of one output row (TMEM lane = this thread's row; warp-collective
// loads, so every lane calls it and only valid rows store): mode 0 BF16 with
// bias, skip and activation; mode 1 FP32, all channels; mode 2 FP32 channel 0.
__device__ __forceinline__ void conv_store(const ConvParams& P, uint32_t trow, bool valid, long long v) {
    if (P.mode == 2) {
        float a[8];
        tmem_ld8(trow, a);
        if (valid) P.out_f[v] = a[0] + (P.bias ? P.bias[0] : 0.f);
        return;
    }
    for (int c0 = 0; c0 < P.cout; c0 += 8) {
        float a[8];
        tmem_ld8(trow + c0, a);
        if (!valid) continue;
        if (P.mode == 1) {
            float4* o = reinterpret_cast<float4*>(P.out_f + v * P.cout + c0);
            o[0] = make_float4(a[0], a[1], a[2], a[3]);
            o[1] = make_float4(a[4], a[5], a[6], a[7]);
        } else {
            uint16_t sk[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            if (P.skip) *reinterpret_cast<uint4*>(sk) = *reinterpret_cast<const uint4*>(P.skip + v * P.cout + c0);
            uint16_t o[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int c = c0 + k;
                float val = a[k];
                if (P.bias && c < P.cout_real) val += P.bias[c];
                if (P.skip) val += bf16_float(sk[k]);
                if (P.relu) val = fmaxf(val, 0.f);
                o[k] = (c < P.cout_real) ? bf16_bits(val) : uint16_t(0);
            }
            *reinterpret_cast<uint4*>(P.out_b + v * P.cout + c0) = *reinterpret_cast<uint4*>(o);
        }
    }
}

// out[v][n] = sum_tap sum_k in[v + off(tap)][k] * w[tap][n][k]
__global__ void __launch_bounds__(kConvM) k_conv(ConvParams P) {
    extern __shared__ __align__(1024) uint8_t sm[];
    const int abytes = kConvM * P.cin * 2;
    const int bbytes = P.cout * P.cin * 2;
    uint8_t* A[2] = {sm, sm + abytes};
    uint8_t* B[2] = {sm + 2 * abytes, sm + 2 * abytes + bbytes};
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + 2 * abytes + 2 * bbytes);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 2);
    __shared__ int abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5;
    const uint32_t ncols = P.cout < 32 ? 32u : uint32_t(P.cout);
    if (tid == 0) {
        abort_flag = 0;
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(tslot, ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;

    const long long v = (long long)blockIdx.x * kConvM + tid;
    const bool valid = v < P.nvox;
    int x = 0, y = 0, z = 0;
    if (valid) {
        z = int(v % P.nz);
        const long long t = v / P.nz;
        y = int(t % P.ny);
        x = int(t / P.ny);
    }
    const int kc = P.cin / 8;             // 16-byte chunks per A/B row
    const uint32_t sbo = uint32_t(kc) * 128;
    const uint32_t idesc = idesc_bf16(kConvM, P.cout, 0, 0);
    int last_tap = -1;
    for (int tap = 0; tap < kNetTaps; ++tap) {
        const int s = tap & 1;
        if (tap >= 2 && !mbar_wait(&bar[s], unsigned((tap - 2) >> 1) & 1u)) abort_flag = 1;
        int dx, dy, dz;
        tap_offset(tap, dx, dy, dz);
        const int xx = x + dx, yy = y + dy, zz = z + dz;
        const bool in = valid && xx >= 0 && xx < P.nx && yy >= 0 && yy < P.ny && zz >= 0 && zz < P.nz;
        const uint4* src = reinterpret_cast<const uint4*>(P.in + (((long long)xx * P.ny + yy) * P.nz + zz) * P.cin);
        uint8_t* arow = A[s] + (tid >> 3) * sbo + (tid & 7) * 16;
        for (int c = 0; c < kc; ++c) {
            const uint4 val = in ? src[c] : make_uint4(0u, 0u, 0u, 0u);
            *reinterpret_cast<uint4*>(arow + c * 128) = val;
        }
        const uint4* wsrc = reinterpret_cast<const uint4*>(P.w + (long long)tap * P.cout * P.cin);
        for (int i = tid; i < bbytes / 16; i += kConvM) reinterpret_cast<uint4*>(B[s])[i] = wsrc[i];
        fence_async_smem();
        __syncthreads();
        if (abort_flag) break;
        if (tid == 0) {
            tc_fence_after();
            const uint32_t a0 = smem_u32(A[s]), b0 = smem_u32(B[s]);
            for (int k = 0; k < P.cin / 16; ++k)
                umma_bf16(tmem, sdesc(a0 + k * 256, 128, sbo), sdesc(b0 + k * 256, 128, sbo), idesc,
                          (tap > 0 || k > 0) ? 1u : 0u);
            umma_commit(&bar[s]);
        }
        last_tap = tap;
    }
    bool ok = !abort_flag;
    if (last_tap >= 0 && !mbar_wait(&bar[last_tap & 1], unsigned(last_tap >> 1) & 1u)) ok = false;
    tc_fence_after();
    __syncwarp();
    // tcgen05.ld is warp-collective: every lane loads, only valid rows store
    if (ok) {
        conv_store(P, tmem + (uint32_t(warp * 32) << 16), valid, v);
    } else if (!ok && valid) {
        // keep the tensor well defined after a timeout
        if (P.mode == 2) P.out_f[v] = 0.f;
    }
    if (!ok && tid == 0 && atomicExch(&P.status->timeout, 1) == 0) {
        P.status->pad[0] = 1;  // kernel: convolution
        P.status->pad[1] = last_tap;
        P.status->pad[2] = int(blockIdx.x);
    }
    tc_fence_before();
    __syncthreads();
    __syncwarp();
    if (warp == 0) tmem_dealloc(tmem, ncols);
}

// ------------------------------------------------------ brick convolution
// The same convolution with the 27 taps reading one staged input brick
// instead of 27 gathers (every layer whose weights and brick fit in shared
// memory).
// An output tile is 128 voxels: one x plane, 16 y rows, 8 z (TMEM lane /
// A row r = (y - y0) * 8 + (z - z0)).  Its input brick, grown by one voxel
// (3 x 18 x 10), sits in shared memory as one plane per 8-channel chunk with
// z fastest, so for any tap the 8 z of a y row are one contiguous 8 x 16-byte
// core matrix: the tap's A operand is the brick at offset (dx, dy, dz), with
// M-direction stride one brick row (160 bytes) and K-direction stride one
// plane.  Each plane is one TMA box {8 channels, 10 z, 18 y, 3 x} of the
// channels-last activations (a 4D tensor map, channels innermost), which
// reads zeros outside the grid: the convolution's zero padding.
//
// CTAs are persistent, keep all 27 weight tiles resident and run their tiles
// as a warp-specialised pipeline over two TMEM accumulators: warp 4 (one
// lane) loads the bricks and issues each tile's MMAs (compile-time
// descriptor offsets from two bases); warps 0-3 drain the accumulators, each
// its 32 TMEM lanes.  They hand over through mbarriers only: a brick has
// landed, a tile's MMAs are done, an accumulator is drained.  Where shared
// memory holds two bricks, tile i + 1's brick loads while tile i's MMAs run.
constexpr int kBrX = 3, kBrY = 18, kBrZ = 10;
constexpr int kBrVox = kBrX * kBrY * kBrZ;  // 540
constexpr int kBrBox = kBrVox * 16;         // bytes of one 8-channel plane (one TMA box)
constexpr int kBrPlane = 68 * 128;          // plane stride: the box rounded up to 128 bytes
constexpr size_t kBrickSmemMax = 227 * 1024;
constexpr int kBrBars = 64;                 // six mbarriers, the TMEM address slot and the abort flag
constexpr int kBrThreads = 160;             // warps 0-3 drain, warp 4 produces

// Shared-memory bytes of the brick kernel for one layer with `stages` bricks.
__host__ __device__ constexpr size_t brick_smem_bytes(int cin, int cout, int stages) {
    return size_t(27) * cout * cin * 2 + size_t(stages) * (cin / 8) * kBrPlane + kBrBars;
}

__device__ __forceinline__ void brick_tile(const ConvParams& P, long long t, int tyn, int tzn, int& x0, int& y0,
                                           int& z0) {
    const long long tt = P.tiles ? (long long)P.tiles[t] : t;
    const int tzi = int(tt % tzn);
    const long long rest = tt / tzn;
    y0 = int(rest % tyn) * 16;
    x0 = int(rest / tyn);
    z0 = tzi * 8;
}

// one thread: the kc planes of tile t's brick into buf
__device__ __forceinline__ void brick_issue(const CUtensorMap* tin, const ConvParams& P, long long t, int tyn, int tzn,
                                            int kc, uint8_t* buf, uint64_t* bar) {
    int x0, y0, z0;
    brick_tile(P, t, tyn, tzn, x0, y0, z0);
    bar_expect_tx(bar, uint32_t(kc * kBrBox));
    for (int c = 0; c < kc; ++c) tma_load_box4(buf + c * kBrPlane, tin, c * 8, z0 - 1, y0 - 1, x0 - 1, bar);
}

// one thread: the 27 x CIN/16 MMAs of one tile, accumulating into acc
template <int CIN, int COUT>
__device__ __forceinline__ void brick_mmas(uint32_t acc, uint32_t a_stage, uint32_t b0) {
    constexpr int KC = CIN / 8;
    constexpr uint32_t idesc = idesc_bf16(kConvM, COUT, 0, 0);
    const uint64_t ad0 = sdesc(a_stage, kBrPlane, kBrZ * 16);
    const uint64_t bd0 = sdesc(b0, 128, uint32_t(KC) * 128);
#pragma unroll
    for (int tap = 0; tap < kNetTaps; ++tap) {
        const int dx = tap / 9, dy = (tap / 3) % 3, dz = tap % 3;  // offsets + 1
        const uint64_t aoff = uint64_t(((dx * kBrY + dy) * kBrZ + dz) * 16) >> 4;
#pragma unroll
        for (int k = 0; k < CIN / 16; ++k)
            umma_bf16(acc, ad0 + aoff + (uint64_t(2 * k * kBrPlane) >> 4),
                      bd0 + (uint64_t(tap * COUT * CIN * 2 + k * 256) >> 4), idesc, (tap > 0 || k > 0) ? 1u : 0u);
    }
}

// Epilogue of one output row (TMEM lane = this thread's row; the loads are
// warp-collective, so every lane calls it and only valid rows store), the
// arithmetic of conv_store: mode 0 BF16 with bias, skip (sk, loaded ahead)
// and activation; mode 1 FP32, all channels; mode 2 FP32 channel 0.
template <int COUT>
__device__ __forceinline__ void brick_store(const ConvParams& P, uint32_t trow, bool valid, long long v,
                                            const uint4 (&sk)[COUT / 8]) {
    if (P.mode == 2) {
        float a[8];
        tmem_ld8(trow, a);
        if (valid) P.out_f[v] = a[0] + (P.bias ? P.bias[0] : 0.f);
        return;
    }
#pragma unroll
    for (int q = 0; q < COUT / 8; ++q) {
        const int c0 = q * 8;
        float a[8];
        tmem_ld8(trow + c0, a);
        if (!valid) continue;
        if (P.mode == 1) {
            float4* o = reinterpret_cast<float4*>(P.out_f + v * COUT + c0);
            o[0] = make_float4(a[0], a[1], a[2], a[3]);
            o[1] = make_float4(a[4], a[5], a[6], a[7]);
        } else {
            uint16_t s8[8];
            *reinterpret_cast<uint4*>(s8) = sk[q];
            uint16_t o[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int c = c0 + k;
                float val = a[k];
                if (P.bias && c < P.cout_real) val += P.bias[c];
                if (P.skip) val += bf16_float(s8[k]);
                if (P.relu) val = fmaxf(val, 0.f);
                o[k] = (c < P.cout_real) ? bf16_bits(val) : uint16_t(0);
            }
            *reinterpret_cast<uint4*>(P.out_b + v * COUT + c0) = *reinterpret_cast<uint4*>(o);
        }
    }
}

// Limit of the brick convolution's pipeline waits (200 ms;
// lhi_debug_set_stage_wait_limit lowers it to test the timeout path, 0
// gives up at once).  The waits for a CTA's own copies and MMAs in flight
// before it leaves keep the fixed 200 ms.
__device__ unsigned long long g_net_wait_ns = 200000000ull;

// Bounded wait on a pipeline barrier that also gives up once another warp of
// the CTA has set the abort flag (a wait of its own that timed out).
__device__ __forceinline__ bool brick_wait(uint64_t* bar, unsigned parity, volatile int* abort_flag) {
    const unsigned long long limit = g_net_wait_ns;
    if (limit == 0) return false;
    const uint32_t addr = smem_u32(bar);
    const uint64_t deadline = global_ns() + limit;
    for (;;) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(addr), "r"(parity)
            : "memory");
        if (ok) return true;
        if (*abort_flag || global_ns() > deadline) return false;
    }
}

// Barriers: full[2] (a brick stage has landed), done[2] (an accumulator's
// MMAs completed), empty[2] (an accumulator has been drained: one arrival
// per draining warp).  Tile i of this CTA uses accumulator i & 1 and, with
// two bricks, brick i & 1.
template <int CIN, int COUT>
__global__ void __launch_bounds__(kBrThreads) k_conv_brick(const __grid_constant__ CUtensorMap tin, ConvParams P,
                                                           int stages) {
    extern __shared__ __align__(1024) uint8_t sm[];
    constexpr int KC = CIN / 8;
    constexpr int WBYTES = COUT * CIN * 2;  // one tap's B tile
    constexpr uint32_t NCOLS = COUT < 32 ? 32u : uint32_t(COUT);
    uint8_t* Bs = sm;
    uint8_t* Ab = sm + 27 * WBYTES;  // brick s at Ab + s * KC * kBrPlane
    uint64_t* full = reinterpret_cast<uint64_t*>(Ab + stages * KC * kBrPlane);
    uint64_t* done = full + 2;
    uint64_t* empty = full + 4;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(full + 6);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tslot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int b = 0; b < 2; ++b) {
            mbar_init(&full[b], 1);
            mbar_init(&done[b], 1);
            mbar_init(&empty[b], 4);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(tslot, 2 * NCOLS);
    for (int i = tid; i < 27 * WBYTES / 16; i += kBrThreads)
        reinterpret_cast<uint4*>(Bs)[i] = reinterpret_cast<const uint4*>(P.w)[i];
    fence_async_smem();  // the weight tiles (generic stores) before the tensor cores read them
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    const int tyn = (P.ny + 15) / 16, tzn = (P.nz + 7) / 8;
    const long long ntiles = P.tiles ? (long long)*P.ntiles : (long long)P.nx * tyn * tzn;
    const long long G = gridDim.x;
    const int nmine = (long long)blockIdx.x < ntiles ? int((ntiles - 1 - blockIdx.x) / G) + 1 : 0;
    if (warp == 4) {
        // ---- producer (one lane)
        if (lane == 0 && nmine > 0) {
            bool pending[2] = {false, false};  // a brick load in flight, not yet waited for
            unsigned use[2] = {0u, 0u};        // completed waits per brick barrier: its next phase's parity
            int last_commit = -1;
            bool ok = true;
            auto brick_buf = [&](int s) { return Ab + s * KC * kBrPlane; };
            brick_issue(&tin, P, blockIdx.x, tyn, tzn, KC, brick_buf(0), &full[0]);
            pending[0] = true;
            for (int i = 0; i < nmine; ++i) {
                const long long t = blockIdx.x + (long long)i * G;
                const int s = stages == 2 ? (i & 1) : 0, b = i & 1;
                if (stages == 1 && i > 0) {
                    // the one brick was read by tile i - 1's MMAs
                    if (!(ok = brick_wait(&done[(i - 1) & 1], unsigned((i - 1) >> 1) & 1u, abort_flag))) break;
                    brick_issue(&tin, P, t, tyn, tzn, KC, brick_buf(0), &full[0]);
                    pending[0] = true;
                }
                if (!(ok = brick_wait(&full[s], use[s] & 1u, abort_flag))) break;
                pending[s] = false;
                ++use[s];
                // accumulator b was last drained after tile i - 2
                if (i >= 2 && !(ok = brick_wait(&empty[b], unsigned((i >> 1) + 1) & 1u, abort_flag))) break;
                tc_fence_after();
                brick_mmas<CIN, COUT>(tmem + uint32_t(b) * NCOLS, smem_u32(brick_buf(s)), smem_u32(Bs));
                umma_commit(&done[b]);
                last_commit = i;
                if (stages == 2 && i + 1 < nmine) {
                    // the other brick was read by tile i - 1's MMAs
                    if (i >= 1 && !(ok = brick_wait(&done[(i - 1) & 1], unsigned((i - 1) >> 1) & 1u, abort_flag)))
                        break;
                    brick_issue(&tin, P, t + G, tyn, tzn, KC, brick_buf(s ^ 1), &full[s ^ 1]);
                    pending[s ^ 1] = true;
                }
            }
            if (!ok) {
                *abort_flag = 1;
                if (atomicExch(&P.status->timeout, 1) == 0) {
                    P.status->pad[0] = 3;  // kernel: brick convolution
                    P.status->pad[2] = int(blockIdx.x);
                }
                // no brick load or MMA of this CTA may still be in flight when it exits
                for (int s2 = 0; s2 < 2; ++s2)
                    if (pending[s2]) mbar_wait(&full[s2], use[s2] & 1u);
                if (last_commit >= 0) mbar_wait(&done[last_commit & 1], unsigned(last_commit >> 1) & 1u);
            }
        }
        __syncwarp();
    } else {
        // ---- drain: warp w reads TMEM lanes 32w .. 32w + 31
        for (int i = 0; i < nmine; ++i) {
            const long long t = blockIdx.x + (long long)i * G;
            const int b = i & 1;
            int x0, y0, z0;
            brick_tile(P, t, tyn, tzn, x0, y0, z0);
            const int y = y0 + (tid >> 3), z = z0 + (tid & 7);
            const bool valid = y < P.ny && z < P.nz;
            const long long v = ((long long)x0 * P.ny + y) * P.nz + z;
            uint4 sk[COUT / 8];
#pragma unroll
            for (int q = 0; q < COUT / 8; ++q) sk[q] = make_uint4(0u, 0u, 0u, 0u);
            if (valid && P.mode == 0 && P.skip) {  // loaded while the MMAs run
                const uint4* src = reinterpret_cast<const uint4*>(P.skip + v * COUT);
#pragma unroll
                for (int q = 0; q < COUT / 8; ++q) sk[q] = src[q];
            }
            // one decision per warp: the TMEM loads are warp-collective
            if (!__all_sync(0xffffffffu, brick_wait(&done[b], unsigned(i >> 1) & 1u, abort_flag))) {
                if (lane == 0) *abort_flag = 1;
                break;
            }
            tc_fence_after();
            brick_store<COUT>(P, tmem + uint32_t(b) * NCOLS + (uint32_t(warp * 32) << 16), valid, v, sk);
            tc_fence_before();
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&empty[b])) : "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, 2 * NCOLS);
}

// ------------------------------------------------------- weight gradient
constexpr int kWgChunk = 64;        // voxels per MMA batch (K)
constexpr int kWgChunksPerCta = 32;  // at most
constexpr int kWgThreads = 128;     // one per row of D
constexpr int kWgCtas = 4;  // an SM

struct WgradParams {
    const uint16_t* g;   // BF16 gradient at the layer output, COUT channels (padded)
    int cout_real;
    const uint16_t* in;  // BF16 layer input, CIN channels (padded)
    int cin_real;
    int nx, ny, nz;
    long long nvox;
    int chunks;          // chunks per CTA
    float* grad_w;       // packed W[27][cout_real][cin_real] of the layer
    NetStatus* status;
};

// D[(tap, co)][ci] = sum_v g[v - off(tap)][co] * in[v][ci] for the 128 / COUT
// taps of blockIdx.y, over P.chunks chunks of kWgChunk input voxels: the tensor
// core's 128 rows hold as many taps as fit (one tap filled COUT of them and
// read the input again for every tap).  A thread carries one 16-byte piece of
// a voxel's channels, consecutive threads the pieces of one voxel, so that a
// warp's loads fill whole lines; the row blocks lie 128 / (pieces) bytes off
// a multiple of 128, which puts a voxel's pieces on different banks.  The next
// chunk's loads are under way while this one's MMAs run.
// What bounds it: latency of the loads, 16 warps an SM; as four CTAs of 64-voxel
// chunks, which wait for one another less (two of 128: 0.23 ms).  Backward of a
// 64^3 grid: 1.02 ms in six launches of one tap a CTA, 0.20 ms now.
template <int COUT, int CIN> struct WgradTile {
    static constexpr int kTaps = 128 / COUT;                          // taps per CTA
    static constexpr int kA = COUT / 8, kB = CIN / 8;                 // 16-byte pieces of a voxel's channels
    static constexpr int kASbo = (kWgChunk / 8) * 128 + 128 / kA;     // bytes between blocks of 8 rows
    static constexpr int kBSbo = (kWgChunk / 8) * 128 + 128 / kB;
    static constexpr int kABytes = (128 / 8) * kASbo, kBBytes = kB * kBSbo;
    static constexpr int kSmem = 2 * (kABytes + kBBytes) + 32;
};

template <int COUT, int CIN> __global__ void __launch_bounds__(kWgThreads, kWgCtas) k_wgrad(WgradParams P) {
    using T = WgradTile<COUT, CIN>;
    constexpr int kTaps = T::kTaps, kA = T::kA, kB = T::kB;
    constexpr int kAv = kWgThreads / kA, kBv = kWgThreads / kB;  // voxels of one step over the threads
    constexpr int kAn = kWgChunk / kAv, kBn = kWgChunk / kBv;    // steps of a chunk
    extern __shared__ __align__(1024) uint8_t sm[];
    uint8_t* A[2] = {sm, sm + T::kABytes};
    uint8_t* B[2] = {sm + 2 * T::kABytes, sm + 2 * T::kABytes + T::kBBytes};
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + 2 * (T::kABytes + T::kBBytes));
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 2);
    bool ok = true;
    const int tid = threadIdx.x, warp = tid >> 5;
    constexpr uint32_t ncols = CIN < 32 ? 32u : uint32_t(CIN);
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(tslot, ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    const int tap0 = blockIdx.y * kTaps;
    // MN-major layout: element (m, k) at (m / 8) * SBO + (k / 8) * 128 + (k % 8) * 16 + (m % 8) * 2
    const uint32_t idesc = idesc_bf16(128, CIN, 1, 1);
    const long long vbase = (long long)blockIdx.x * P.chunks * kWgChunk;
    uint4 ra[kAn][kTaps], rb[kBn];
    auto fetch = [&](int ch) {  // this thread's pieces of chunk ch
        const long long v0 = ch < P.chunks ? vbase + (long long)ch * kWgChunk : P.nvox;
#pragma unroll
        for (int n = 0; n < kBn; ++n) {
            const long long v = v0 + n * kBv + tid / kB;
            rb[n] = v < P.nvox ? reinterpret_cast<const uint4*>(P.in + v * CIN)[tid % kB] : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int n = 0; n < kAn; ++n) {
            const long long v = v0 + n * kAv + tid / kA;
            int x, y, z;
            idx3(v, P.ny, P.nz, x, y, z);
            // bit d + 1: coordinate - d lies in the grid
            const unsigned mx = unsigned(x + 1 < P.nx) | 2u | unsigned(x > 0) << 2;
            const unsigned my = unsigned(y + 1 < P.ny) | 2u | unsigned(y > 0) << 2;
            const unsigned mz = unsigned(z + 1 < P.nz) | 2u | unsigned(z > 0) << 2;
            const uint4* g = reinterpret_cast<const uint4*>(P.g) + v * kA + tid % kA;
#pragma unroll
            for (int k = 0; k < kTaps; ++k) {
                const int tap = tap0 + k;
                int dx, dy, dz;
                tap_offset(tap, dx, dy, dz);
                const bool in = v < P.nvox && tap < kNetTaps && (mx >> (dx + 1) & my >> (dy + 1) & mz >> (dz + 1) & 1u);
                ra[n][k] = in ? g[-(((long long)dx * P.ny + dy) * P.nz + dz) * kA] : make_uint4(0u, 0u, 0u, 0u);
            }
        }
    };
    auto koff = [](int k) { return uint32_t(k >> 3) * 128 + uint32_t(k & 7) * 16; };
    fetch(0);
    int issued = 0;
    for (int ch = 0; ch < P.chunks; ++ch) {
        if (vbase + (long long)ch * kWgChunk >= P.nvox) break;
        const int s = ch & 1;
        if (ch >= 2 && !mbar_wait(&bar[s], unsigned((ch - 2) >> 1) & 1u)) ok = false;
#pragma unroll
        for (int n = 0; n < kAn; ++n)
#pragma unroll
            for (int k = 0; k < kTaps; ++k)
                *reinterpret_cast<uint4*>(A[s] + (k * kA + tid % kA) * T::kASbo + koff(n * kAv + tid / kA)) = ra[n][k];
#pragma unroll
        for (int n = 0; n < kBn; ++n)
            *reinterpret_cast<uint4*>(B[s] + (tid % kB) * T::kBSbo + koff(n * kBv + tid / kB)) = rb[n];
        fence_async_smem();
        if (__syncthreads_or(!ok)) {
            ok = false;
            break;
        }
        if (tid == 0) {
            tc_fence_after();
            const uint32_t a0 = smem_u32(A[s]), b0 = smem_u32(B[s]);
            for (int k = 0; k < kWgChunk / 16; ++k)
                umma_bf16(tmem, sdesc(a0 + k * 256, 128, T::kASbo), sdesc(b0 + k * 256, 128, T::kBSbo), idesc,
                          (issued > 0 || k > 0) ? 1u : 0u);
            umma_commit(&bar[s]);
        }
        issued = ch + 1;
        fetch(ch + 1);
    }
    if (issued > 0 && !mbar_wait(&bar[(issued - 1) & 1], unsigned((issued - 1) >> 1) & 1u)) ok = false;
    tc_fence_after();
    ok = __all_sync(0xffffffffu, ok);
    if (ok && issued > 0) {
        // warp w reads the rows of quarter w (TMEM lane = row of D = thread), all columns
        const uint32_t trow = tmem + (uint32_t(warp * 32) << 16);
        const int tap = tap0 + tid / COUT, co = tid % COUT;
        for (int c0 = 0; c0 < CIN; c0 += 8) {
            float a[8];
            tmem_ld8(trow + c0, a);
            if (co < P.cout_real && tap < kNetTaps) {
                float* g = P.grad_w + ((long long)tap * P.cout_real + co) * P.cin_real + c0;
#pragma unroll
                for (int k = 0; k < 8; k += 4)  // cin_real and the layer's offset are multiples of 4
                    if (c0 + k < P.cin_real)
                        atomicAdd(reinterpret_cast<float4*>(g + k), make_float4(a[k], a[k + 1], a[k + 2], a[k + 3]));
            }
        }
    }
    if (!ok && tid == 0 && atomicExch(&P.status->timeout, 1) == 0) {
        P.status->pad[0] = 2;  // kernel: weight gradient
        P.status->pad[1] = issued;
        P.status->pad[2] = int(blockIdx.x);
    }
    tc_fence_before();
    __syncthreads();
    __syncwarp();
    if (warp == 0) tmem_dealloc(tmem, ncols);
}

// One CTA, one 128 x N x K bf16 GEMM through the same descriptors and
// pipeline pieces as the convolutions: D[m][n] = sum_k A[m][k] B[n][k], A and
// B given row-major in global memory (K-major).  Records in status how far
// it got: pad[3] = 1 after TMEM allocation, 2 after the MMAs were issued, 3
// after their commit arrived, 4 after the TMEM read.
__global__ void __launch_bounds__(128) k_umma_selftest(const uint16_t* __restrict__ a, const uint16_t* __restrict__ b,
                                                       int N, int K, float* __restrict__ d, NetStatus* status) {
    __shared__ __align__(1024) uint8_t As[128 * 64 * 2];
    __shared__ __align__(1024) uint8_t Bs[64 * 64 * 2];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tslot;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int kc = K / 8;
    const uint32_t sbo = uint32_t(kc) * 128;
    for (int c = 0; c < kc; ++c)
        *reinterpret_cast<uint4*>(As + (tid >> 3) * sbo + (tid & 7) * 16 + c * 128) =
            reinterpret_cast<const uint4*>(a + (long long)tid * K)[c];
    if (tid < N)
        for (int c = 0; c < kc; ++c)
            *reinterpret_cast<uint4*>(Bs + (tid >> 3) * sbo + (tid & 7) * 16 + c * 128) =
                reinterpret_cast<const uint4*>(b + (long long)tid * K)[c];
    if (tid == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(&tslot, 64);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tslot;
    if (tid == 0) {
        status->pad[3] = 1;
        const uint32_t idesc = idesc_bf16(128, N, 0, 0);
        for (int k = 0; k < K / 16; ++k)
            umma_bf16(tmem, sdesc(smem_u32(As) + k * 256, 128, sbo), sdesc(smem_u32(Bs) + k * 256, 128, sbo), idesc,
                      k > 0 ? 1u : 0u);
        umma_commit(&bar);
        status->pad[3] = 2;
    }
    const bool ok = mbar_wait(&bar, 0);
    if (tid == 0 && ok) status->pad[3] = 3;
    tc_fence_after();
    __syncwarp();
    if (ok) {
        for (int c0 = 0; c0 < N; c0 += 8) {
            float v[8];
            tmem_ld8(tmem + (uint32_t(warp * 32) << 16) + c0, v);
            for (int k = 0; k < 8; ++k) d[(long long)tid * N + c0 + k] = v[k];
        }
        if (tid == 0) status->pad[3] = 4;
    } else if (tid == 0) {
        atomicExch(&status->timeout, 1);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 64);
}

// ------------------------------------------------------------ elementwise
__device__ __forceinline__ void dec3(long long v, int ny, int nz, int& x, int& y, int& z) {
    z = int(v % nz);
    const long long t = v / nz;
    y = int(t % ny);
    x = int(t / ny);
}

// sum r^2 and count over fluid cells -> s = sqrt(sum / count) (1 if empty)
__global__ void k_net_scale(const float* __restrict__ r, const uint8_t* __restrict__ type, long long n,
                            double* __restrict__ partials, unsigned* __restrict__ counter, float* __restrict__ scale) {
    double v[2] = {0.0, 0.0};
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        if (type[i] != 0) {
            v[0] += double(r[i]) * double(r[i]);
            v[1] += 1.0;
        }
    double tot[2];
    if (!grid_sum_last<2>(v, partials, counter, tot)) return;
    const double s = (tot[1] > 0 && tot[0] > 0) ? sqrt(tot[0] / tot[1]) : 1.0;
    *scale = float(s);
}

// Input channels, all linear in r so that M(a r) = a M(r) for a > 0 and
// M(0) = 0: [r/s, r/s on cells next to air, r/s on cells next to a solid
// (or the domain edge), 0], on cells with type != 0.
__device__ __forceinline__ void net_input_voxel(const float* __restrict__ r, const uint8_t* __restrict__ type,
                                                const uint8_t* __restrict__ solid, int nx, int ny, int nz,
                                                const float* __restrict__ scale, uint16_t* __restrict__ a0,
                                                long long v) {
    const bool fl = type[v] != 0;
    bool air = false, sol = false;
    if (fl) {
        int x, y, z;
        z = int(v % nz);
        const long long t = v / nz;
        y = int(t % ny);
        x = int(t / ny);
        const int dx[6] = {1, -1, 0, 0, 0, 0}, dy[6] = {0, 0, 1, -1, 0, 0}, dz[6] = {0, 0, 0, 0, 1, -1};
        for (int k = 0; k < 6; ++k) {
            const int xx = x + dx[k], yy = y + dy[k], zz = z + dz[k];
            if (xx < 0 || xx >= nx || yy < 0 || yy >= ny || zz < 0 || zz >= nz) {
                sol = true;
                continue;
            }
            const long long u = ((long long)xx * ny + yy) * nz + zz;
            if (solid && solid[u]) sol = true;
            else if (type[u] == 0) air = true;
        }
    }
    const float rh = fl ? r[v] / *scale : 0.f;
    uint16_t o[16] = {};
    o[0] = bf16_bits(rh);
    o[1] = bf16_bits(air ? rh : 0.f);
    o[2] = bf16_bits(sol ? rh : 0.f);
    uint4* dst = reinterpret_cast<uint4*>(a0 + v * 16);
    dst[0] = reinterpret_cast<uint4*>(o)[0];
    dst[1] = reinterpret_cast<uint4*>(o)[1];
}

__global__ void k_net_input(const float* __restrict__ r, const uint8_t* __restrict__ type,
                            const uint8_t* __restrict__ solid, int nx, int ny, int nz, const float* __restrict__ scale,
                            uint16_t* __restrict__ a0) {
    const long long n = (long long)nx * ny * nz;
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    net_input_voxel(r, type, solid, nx, ny, nz, scale, a0, v);
}

// The voxel of this thread in tile u of a brick-tile list (one x plane,
// 16 y, 8 z; thread = (y - y0) * 8 + (z - z0), as the convolution's rows);
// false past the grid's edge.
__device__ __forceinline__ bool list_voxel(const int32_t* __restrict__ list, int u, int ny, int nz, int& x, int& y,
                                           int& z) {
    const int tyn = (ny + 15) / 16, tzn = (nz + 7) / 8;
    const long long tt = list[u];
    const int tzi = int(tt % tzn);
    const long long rest = tt / tzn;
    x = int(rest / tyn);
    y = int(rest % tyn) * 16 + (threadIdx.x >> 3);
    z = tzi * 8 + (threadIdx.x & 7);
    return y < ny && z < nz;
}

// k_net_input on the voxels of the listed tiles (128 threads per block)
__global__ void __launch_bounds__(128) k_net_input_tiles(const float* __restrict__ r, const uint8_t* __restrict__ type,
                                                         const uint8_t* __restrict__ solid, int nx, int ny, int nz,
                                                         const float* __restrict__ scale, uint16_t* __restrict__ a0,
                                                         const int32_t* __restrict__ list, const int* __restrict__ count) {
    const int n = *count;
    for (int u = blockIdx.x; u < n; u += gridDim.x) {
        int x, y, z;
        if (list_voxel(list, u, ny, nz, x, y, z)) net_input_voxel(r, type, solid, nx, ny, nz, scale, a0, ((long long)x * ny + y) * nz + z);
    }
}

// k_pool on the coarse voxels of the listed tiles: the same per-channel sums
// (children in order, FP32) for the voxel's C channels
__global__ void __launch_bounds__(128) k_pool_tiles(const uint16_t* __restrict__ fine, int fny, int fnz,
                                                    uint16_t* __restrict__ coarse, int cny, int cnz, int C,
                                                    const int32_t* __restrict__ list, const int* __restrict__ count) {
    const int n = *count;
    for (int u = blockIdx.x; u < n; u += gridDim.x) {
        int x, y, z;
        if (!list_voxel(list, u, cny, cnz, x, y, z)) continue;
        const long long v = ((long long)x * cny + y) * cnz + z;
        for (int q = 0; q < C / 8; ++q) {
            float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const long long f = ((long long)(2 * x + (k >> 2)) * fny + (2 * y + ((k >> 1) & 1))) * fnz + (2 * z + (k & 1));
                uint16_t c8[8];
                *reinterpret_cast<uint4*>(c8) = reinterpret_cast<const uint4*>(fine + f * C)[q];
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j] += bf16_float(c8[j]);
            }
            uint16_t o[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = bf16_bits(acc[j] * 0.125f);
            reinterpret_cast<uint4*>(coarse + v * C)[q] = *reinterpret_cast<uint4*>(o);
        }
    }
}

// k_upsample on the fine voxels of the listed tiles
__global__ void __launch_bounds__(128) k_upsample_tiles(const uint16_t* __restrict__ coarse, int cnx, int cny, int cnz,
                                                        uint16_t* __restrict__ fine, int fny, int fnz, int C,
                                                        const int32_t* __restrict__ list, const int* __restrict__ count) {
    const int n = *count;
    for (int u = blockIdx.x; u < n; u += gridDim.x) {
        int x, y, z;
        if (!list_voxel(list, u, fny, fnz, x, y, z)) continue;
        const int px = x >> 1, py = y >> 1, pz = z >> 1;
        const bool in = px < cnx && py < cny && pz < cnz;
        const uint4* src = reinterpret_cast<const uint4*>(coarse + (((long long)px * cny + py) * cnz + pz) * C);
        uint4* dst = reinterpret_cast<uint4*>(fine + (((long long)x * fny + y) * fnz + z) * C);
        for (int q = 0; q < C / 8; ++q) dst[q] = in ? src[q] : make_uint4(0u, 0u, 0u, 0u);
    }
}

// Eight channels of a voxel.  The layers' channel counts are multiples of 8, so
// that a thread of the kernels below moves whole 16-byte pieces (32 bytes of
// FP32) and finds its voxel once for all of them.  One channel a thread, the
// nine launches of a forward and backward at 64^3 took 87 us, 47 now.
struct Ch8 {
    float v[8];
};
__device__ __forceinline__ Ch8 ch8_load(const uint16_t* p, long long piece) {
    const uint4 w = reinterpret_cast<const uint4*>(p)[piece];
    const unsigned u[4] = {w.x, w.y, w.z, w.w};
    Ch8 r;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        r.v[2 * k] = bf16_float(uint16_t(u[k]));
        r.v[2 * k + 1] = bf16_float(uint16_t(u[k] >> 16));
    }
    return r;
}
__device__ __forceinline__ Ch8 ch8_load(const float* p, long long piece) {
    const float4 a = reinterpret_cast<const float4*>(p)[2 * piece], b = reinterpret_cast<const float4*>(p)[2 * piece + 1];
    return {{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
}
__device__ __forceinline__ void ch8_store(uint16_t* p, long long piece, const Ch8& r) {
    unsigned u[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) u[k] = unsigned(bf16_bits(r.v[2 * k])) | unsigned(bf16_bits(r.v[2 * k + 1])) << 16;
    reinterpret_cast<uint4*>(p)[piece] = make_uint4(u[0], u[1], u[2], u[3]);
}
__device__ __forceinline__ void ch8_store(float* p, long long piece, const Ch8& r) {
    reinterpret_cast<float4*>(p)[2 * piece] = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
    reinterpret_cast<float4*>(p)[2 * piece + 1] = make_float4(r.v[4], r.v[5], r.v[6], r.v[7]);
}
// sum of the 8 children's channels, children in (x, y, z) order
template <typename T>
__device__ __forceinline__ Ch8 ch8_children(const T* fine, int x, int y, int z, int fny, int fnz, int q, int piece) {
    Ch8 c[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const long long f = ((long long)(2 * x + (k >> 2)) * fny + (2 * y + ((k >> 1) & 1))) * fnz + (2 * z + (k & 1));
        c[k] = ch8_load(fine, f * q + piece);
    }
    Ch8 acc = {};
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc.v[j] += c[k].v[j];
    return acc;
}

// coarse[v][c] = bf16(0.125 * sum of the 8 children)
__global__ void k_pool(const uint16_t* __restrict__ fine, int fny, int fnz, uint16_t* __restrict__ coarse, int cnx,
                       int cny, int cnz, int C) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int q = C / 8;
    if (i >= (long long)cnx * cny * cnz * q) return;
    const long long v = i / q;
    int x, y, z;
    idx3(v, cny, cnz, x, y, z);
    Ch8 acc = ch8_children(fine, x, y, z, fny, fnz, q, int(i - v * q));
#pragma unroll
    for (int j = 0; j < 8; ++j) acc.v[j] *= 0.125f;
    ch8_store(coarse, i, acc);
}

// fine[v][c] = coarse[parent(v)][c] (0 beyond 2 * coarse extent)
// fine voxel (x, y, z) = coarse voxel (x/2, y/2, z/2), 0 past the coarse
// grid.  One thread per fine voxel and 8-channel (16-byte) chunk; C is a
// multiple of 8 and every voxel's channels start on a 16-byte boundary.
__global__ void k_upsample(const uint16_t* __restrict__ coarse, int cnx, int cny, int cnz, uint16_t* __restrict__ fine,
                           int fnx, int fny, int fnz, int C) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned q = unsigned(C) / 8;
    if (i >= unsigned(fnx) * unsigned(fny) * unsigned(fnz) * q) return;
    const unsigned v = i / q, ch = i - v * q;
    int x, y, z;
    idx3(v, fny, fnz, x, y, z);
    const int px = x >> 1, py = y >> 1, pz = z >> 1;
    uint4 val = make_uint4(0u, 0u, 0u, 0u);
    if (px < cnx && py < cny && pz < cnz)
        val = reinterpret_cast<const uint4*>(coarse)[((unsigned(px) * cny + py) * cnz + pz) * q + ch];
    reinterpret_cast<uint4*>(fine)[i] = val;
}

// dcoarse[v][c] = sum of the 8 children's dfine (FP32)
__global__ void k_sum_children(const float* __restrict__ fine, int fny, int fnz, float* __restrict__ coarse, int cnx,
                               int cny, int cnz, int C) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int q = C / 8;
    if (i >= (long long)cnx * cny * cnz * q) return;
    const long long v = i / q;
    int x, y, z;
    idx3(v, cny, cnz, x, y, z);
    ch8_store(coarse, i, ch8_children(fine, x, y, z, fny, fnz, q, int(i - v * q)));
}

// g = bf16(d * relu'(u)), or bf16(d) for the linear network; n in eights of channels
__global__ void k_relu_grad(const float* __restrict__ d, const uint16_t* __restrict__ u, long long n, int relu,
                            uint16_t* __restrict__ g) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Ch8 r = ch8_load(d, i);
    if (relu) {
        const Ch8 w = ch8_load(u, i);
#pragma unroll
        for (int j = 0; j < 8; ++j) r.v[j] = w.v[j] > 0.f ? r.v[j] : 0.f;
    }
    ch8_store(g, i, r);
}

// g = bf16((skip + 0.125 * dcoarse[parent]) * relu'(u)) at a fine level
__global__ void k_relu_grad_unpool(const uint16_t* __restrict__ skip, const float* __restrict__ dcoarse, int cnx, int cny,
                                   int cnz, const uint16_t* __restrict__ u, int fnx, int fny, int fnz, int C,
                                   int relu, uint16_t* __restrict__ g) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int q = C / 8;
    if (i >= (long long)fnx * fny * fnz * q) return;
    const long long v = i / q;
    int x, y, z;
    idx3(v, fny, fnz, x, y, z);
    const int px = x >> 1, py = y >> 1, pz = z >> 1;
    Ch8 r = ch8_load(skip, i);
    if (px < cnx && py < cny && pz < cnz) {
        const Ch8 c = ch8_load(dcoarse, (((long long)px * cny + py) * cnz + pz) * q + (i - v * q));
#pragma unroll
        for (int j = 0; j < 8; ++j) r.v[j] = fmaf(0.125f, c.v[j], r.v[j]);
    }
    if (relu) {
        const Ch8 w = ch8_load(u, i);
#pragma unroll
        for (int j = 0; j < 8; ++j) r.v[j] = w.v[j] > 0.f ? r.v[j] : 0.f;
    }
    ch8_store(g, i, r);
}

// z = s * y on fluid cells
__global__ void k_net_output(const float* __restrict__ y, const uint8_t* __restrict__ type, long long n,
                             const float* __restrict__ scale, float* __restrict__ z) {
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    z[v] = (type[v] != 0) ? y[v] * *scale : 0.f;
}

// g5[v] = [bf16(s * dz * fluid), 0, ..., 0]
__global__ void k_net_dy(const float* __restrict__ dz, const uint8_t* __restrict__ type, long long n,
                         const float* __restrict__ scale, uint16_t* __restrict__ g5) {
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    uint16_t o[16] = {};
    o[0] = bf16_bits(type[v] != 0 ? dz[v] * *scale : 0.f);
    uint4* dst = reinterpret_cast<uint4*>(g5 + v * 16);
    dst[0] = reinterpret_cast<uint4*>(o)[0];
    dst[1] = reinterpret_cast<uint4*>(o)[1];
}

// B tiles of one layer: forward [tap][n = cout_pad][k = cin_pad] holding
// W[tap][n][k]; backward [tap][n = cin_pad][k = cout_pad] holding
// W[26 - tap][k][n].  K-major core-matrix layout, zero padding.
__global__ void k_format_weights(const float* __restrict__ w, int cout, int cin, uint16_t* __restrict__ fwd,
                                 uint16_t* __restrict__ bwd) {
    const int cop = pad16(cout), cip = pad16(cin);
    const long long per_tap = (long long)cop * cip;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= per_tap * kNetTaps) return;
    const int tap = int(i / per_tap);
    const int rem = int(i % per_tap);
    {  // forward element (n, k)
        const int n = rem / cip, k = rem % cip;
        const float val = (n < cout && k < cin) ? w[((long long)tap * cout + n) * cin + k] : 0.f;
        const long long off = (long long)(n / 8) * (cip / 8) * 64 + (k / 8) * 64 + (n % 8) * 8 + (k % 8);
        fwd[tap * per_tap + off] = bf16_bits(val);
    }
    if (bwd) {  // backward element (n = ci, k = co)
        const int n = rem / cop, k = rem % cop;
        const float val = (n < cin && k < cout) ? w[((long long)(kNetTaps - 1 - tap) * cout + k) * cin + n] : 0.f;
        const long long off = (long long)(n / 8) * (cop / 8) * 64 + (k / 8) * 64 + (n % 8) * 8 + (k % 8);
        bwd[tap * per_tap + off] = bf16_bits(val);
    }
}

__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       long long n, float lr, float b1, float b2, float eps, float c1, float c2) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

unsigned nb(long long n, int t = 256) { return unsigned(std::max<long long>(1, (n + t - 1) / t)); }


// ------------------------------------------------- sparse evaluation plan
// Byte masks of the voxels each convolution's output must be right on, and
// from them the output tiles (the brick kernel's 128-voxel tiles) to
// evaluate.  Voxels outside these sets may hold stale values: every value a
// needed voxel reads (its 27 neighbours, its pooled children, its upsampled
// parent, its skip input) is itself needed, and the tensor-core product of
// a tile row reads that row's inputs only.
__global__ void k_mask_type(const uint8_t* __restrict__ type, long long n, uint8_t* __restrict__ m) {
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v < n) m[v] = type[v] != 0;
}

// out = in dilated by one voxel along z (axis 0) or along x and y (axis 1)
__global__ void k_mask_dilate(const uint8_t* __restrict__ in, int nx, int ny, int nz, int axis,
                              uint8_t* __restrict__ out) {
    const long long n = (long long)nx * ny * nz;
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    int x, y, z;
    dec3(v, ny, nz, x, y, z);
    uint8_t o = 0;
    if (axis == 0) {
        o = in[v];
        if (z > 0) o |= in[v - 1];
        if (z + 1 < nz) o |= in[v + 1];
    } else {
        for (int dx = -1; dx <= 1; ++dx)
            for (int dy = -1; dy <= 1; ++dy) {
                const int xx = x + dx, yy = y + dy;
                if (xx >= 0 && xx < nx && yy >= 0 && yy < ny) o |= in[((long long)xx * ny + yy) * nz + z];
            }
    }
    out[v] = o;
}

// k_mask_dilate over 4-voxel words along z (nz a multiple of 4, so a word
// never spans two z rows): axis 0 along z, axis 1 along x and y
__global__ void k_mask_dilate4(const uint32_t* __restrict__ in, int nx, int ny, int nzw, int axis,
                               uint32_t* __restrict__ out) {
    const long long n = (long long)nx * ny * nzw;
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    int x, y, zw;
    dec3(v, ny, nzw, x, y, zw);
    uint32_t o;
    if (axis == 0) {
        const uint32_t w = in[v];
        o = w | (w << 8) | (w >> 8);
        if (zw > 0) o |= in[v - 1] >> 24;       // z - 1 of the first voxel
        if (zw + 1 < nzw) o |= in[v + 1] << 24;  // z + 1 of the last voxel
    } else {
        o = 0u;
        for (int dx = -1; dx <= 1; ++dx)
            for (int dy = -1; dy <= 1; ++dy) {
                const int xx = x + dx, yy = y + dy;
                if (xx >= 0 && xx < nx && yy >= 0 && yy < ny) o |= in[((long long)xx * ny + yy) * nzw + zw];
            }
    }
    out[v] = o;
}

// k_mask_tile_flags over 4-voxel words (nz a multiple of 4: a word lies in
// one tile's 8 z)
__global__ void k_mask_tile_flags4(const uint32_t* __restrict__ m, int nx, int ny, int nzw, int nz,
                                   uint8_t* __restrict__ flag) {
    const long long n = (long long)nx * ny * nzw;
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n || !m[v]) return;
    int x, y, zw;
    dec3(v, ny, nzw, x, y, zw);
    const int tyn = (ny + 15) / 16, tzn = (nz + 7) / 8;
    flag[((long long)x * tyn + (y >> 4)) * tzn + (zw >> 1)] = 1;
}

// coarse voxel set if any of its 8 children is (the voxels whose upsampled
// value a needed fine voxel reads)
__global__ void k_mask_up(const uint8_t* __restrict__ fine, int fny, int fnz, int cnx, int cny, int cnz,
                          uint8_t* __restrict__ coarse) {
    const long long n = (long long)cnx * cny * cnz;
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    int x, y, z;
    dec3(v, cny, cnz, x, y, z);
    uint8_t o = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k)
        o |= fine[((long long)(2 * x + (k >> 2)) * fny + (2 * y + ((k >> 1) & 1))) * fnz + (2 * z + (k & 1))];
    coarse[v] = o;
}

// out = other | (fine voxels whose parent is set: the children a needed
// pooled voxel averages)
__global__ void k_mask_down_or(const uint8_t* __restrict__ coarse, int cnx, int cny, int cnz,
                               const uint8_t* __restrict__ other, int fnx, int fny, int fnz, uint8_t* __restrict__ out) {
    const long long n = (long long)fnx * fny * fnz;
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    int x, y, z;
    dec3(v, fny, fnz, x, y, z);
    const int px = x >> 1, py = y >> 1, pz = z >> 1;
    uint8_t o = other[v];
    if (px < cnx && py < cny && pz < cnz) o |= coarse[((long long)px * cny + py) * cnz + pz];
    out[v] = o;
}

// flag[t] = 1 for the brick tiles (x, y / 16, z / 8) holding a set voxel
__global__ void k_mask_tile_flags(const uint8_t* __restrict__ m, int nx, int ny, int nz, uint8_t* __restrict__ flag) {
    const long long n = (long long)nx * ny * nz;
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n || !m[v]) return;
    int x, y, z;
    dec3(v, ny, nz, x, y, z);
    const int tyn = (ny + 15) / 16, tzn = (nz + 7) / 8;
    flag[((long long)x * tyn + (y >> 4)) * tzn + (z >> 3)] = 1;
}

// list of the flagged tiles (in any order) and their count
__global__ void k_mask_tile_list(const uint8_t* __restrict__ flag, long long ntiles, int32_t* __restrict__ list,
                                 int* __restrict__ count) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntiles || !flag[t]) return;
    list[atomicAdd(count, 1)] = int32_t(t);
}

}  // namespace

// ------------------------------------------------------------- host side
LearnedNet::LearnedNet(uint64_t seed) {
    const long long np = net_param_count();
    std::vector<float> w(size_t(np), 0.f);
    std::mt19937_64 rng(seed);
    for (int l = 0; l < kNetLayers; ++l) {
        const long long off = net_param_offset(l);
        const int fan_in = kNetTaps * kNetCin[l];
        const double sd = std::sqrt(2.0 / fan_in) * (l == kNetLayers - 1 ? 0.5 : 1.0);
        std::normal_distribution<double> nd(0.0, sd);
        const long long nw = (long long)kNetTaps * kNetCout[l] * kNetCin[l];
        for (long long i = 0; i < nw; ++i) w[size_t(off + i)] = float(nd(rng));
    }
    LHI_CUDA(cudaMalloc(&w32_, sizeof(float) * np));
    LHI_CUDA(cudaMalloc(&grad_, sizeof(float) * np));
    LHI_CUDA(cudaMalloc(&adam_m_, sizeof(float) * np));
    LHI_CUDA(cudaMalloc(&adam_v_, sizeof(float) * np));
    LHI_CUDA(cudaMemcpy(w32_, w.data(), sizeof(float) * np, cudaMemcpyHostToDevice));
    LHI_CUDA(cudaMemset(grad_, 0, sizeof(float) * np));
    LHI_CUDA(cudaMemset(adam_m_, 0, sizeof(float) * np));
    LHI_CUDA(cudaMemset(adam_v_, 0, sizeof(float) * np));
    long long f = 0;
    for (int l = 0; l < kNetLayers; ++l) {
        wfwd_off_[l] = f;
        wbwd_off_[l] = f;
        f += (long long)kNetTaps * pad16(kNetCout[l]) * pad16(kNetCin[l]);
    }
    LHI_CUDA(cudaMalloc(&wfwd_, sizeof(uint16_t) * f));
    LHI_CUDA(cudaMalloc(&wbwd_, sizeof(uint16_t) * f));
    LHI_CUDA(cudaMalloc(&status_, sizeof(NetStatus)));
    LHI_CUDA(cudaMemset(status_, 0, sizeof(NetStatus)));
    LHI_CUDA(cudaMalloc(&scale_, sizeof(float)));
    LHI_CUDA(cudaMalloc(&red_, sizeof(double) * 2 * 1024));
    LHI_CUDA(cudaMalloc(&counter_, sizeof(unsigned) * 4));
    LHI_CUDA(cudaMemset(counter_, 0, sizeof(unsigned) * 4));
    LHI_CUDA(cudaFuncSetAttribute(k_conv, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024));
}

LearnedNet::~LearnedNet() {
    auto F = [](void* p) {
        if (p) cudaFree(p);
    };
    F(w32_), F(grad_), F(adam_m_), F(adam_v_), F(wfwd_), F(wbwd_), F(status_), F(scale_), F(red_), F(counter_);
}

void LearnedNet::set_params(const float* host) {
    LHI_CUDA(cudaMemcpy(w32_, host, sizeof(float) * net_param_count(), cudaMemcpyHostToDevice));
    wfmt_stale_ = true;
}
void LearnedNet::get_params(float* host) {
    LHI_CUDA(cudaMemcpy(host, w32_, sizeof(float) * net_param_count(), cudaMemcpyDeviceToHost));
}
void LearnedNet::get_grads(float* host, cudaStream_t s) {
    LHI_CUDA(cudaMemcpyAsync(host, grad_, sizeof(float) * net_param_count(), cudaMemcpyDeviceToHost, s));
    LHI_CUDA(cudaStreamSynchronize(s));
}
void LearnedNet::zero_grad(cudaStream_t s) {
    LHI_CUDA(cudaMemsetAsync(grad_, 0, sizeof(float) * net_param_count(), s));
}
int LearnedNet::check_status(cudaStream_t s) {
    NetStatus h{};
    LHI_CUDA(cudaMemcpyAsync(&h, status_, sizeof(h), cudaMemcpyDeviceToHost, s));
    LHI_CUDA(cudaStreamSynchronize(s));
    if (h.timeout) {
        last_timeout_[0] = h.pad[0];
        last_timeout_[1] = h.pad[1];
        last_timeout_[2] = h.pad[2];
        // reported once: the next call starts from a clear status
        LHI_CUDA(cudaMemsetAsync(status_, 0, sizeof(NetStatus), s));
        LHI_CUDA(cudaStreamSynchronize(s));
    }
    return h.timeout ? LHI_E_TIMEOUT : LHI_OK;
}

void set_net_wait_limit_ns(unsigned long long ns) {
    LHI_CUDA(cudaMemcpyToSymbol(g_net_wait_ns, &ns, sizeof(ns)));
}

void LearnedNet::ensure(const int dims[3]) {
    for (int a = 0; a < 3; ++a)
        if (dims[a] < 4) throw std::invalid_argument("learned preconditioner: grid below 4 cells on an axis");
    if (layer_mem_.fits(dims)) return;
    const NetLevels n = net_levels(dims);
    b_ = NetBuffers();  // no grid's, until every buffer is there
    layer_mem_.fit(dims, layer_bytes(n));
    NetBuffers b;
    size_t m = 0;
    for (uint16_t** p : {&b.a0, &b.h0, &b.p0, &b.h1, &b.p1, &b.h2, &b.q1, &b.u1, &b.q0, &b.u0})
        *p = layer_mem_.at<uint16_t>(m++);
    b.y = layer_mem_.at<float>(m++);
    for (uint16_t*& p : b.g) p = layer_mem_.at<uint16_t>(m++);
    b.dx = layer_mem_.at<float>(m++);
    b.acc = layer_mem_.at<float>(m);
    for (int l = 0; l < 3; ++l) {
        for (int a = 0; a < 3; ++a) b.dims[l][a] = n.d[l][a];
        b.vox[l] = n.vox(l);
    }
    b_ = b;
}

void LearnedNet::reserve(const int dims[3], bool plan) {
    ensure(dims);
    if (!plan) return;
    if (!plan_mem_.holds(plan_bytes(net_levels(dims)))) plan_type_ = nullptr;  // the lists go
    plan_mem_.fit(plan_bytes(net_levels(dims)));
}

void LearnedNet::format_weights(cudaStream_t s) {
    for (int l = 0; l < kNetLayers; ++l) {
        const long long n = (long long)kNetTaps * pad16(kNetCout[l]) * pad16(kNetCin[l]);
        k_format_weights<<<nb(n), 256, 0, s>>>(w32_ + net_param_offset(l), kNetCout[l], kNetCin[l], wfwd_ + wfwd_off_[l],
                                               l == 0 ? nullptr : wbwd_ + wbwd_off_[l]);
        LHI_LAUNCH_CHECK();
    }
    wfmt_stale_ = false;
}

namespace {
template <int CIN, int COUT>
void launch_brick_t(const CUtensorMap& tin, const ConvParams& P, int stages, unsigned grid, size_t smem, cudaStream_t s) {
    static bool attr = false;
    if (!attr) {
        LHI_CUDA(cudaFuncSetAttribute(k_conv_brick<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      int(kBrickSmemMax)));
        attr = true;
    }
    k_conv_brick<CIN, COUT><<<grid, kBrThreads, smem, s>>>(tin, P, stages);
    LHI_LAUNCH_CHECK();
}

// The brick kernel's instances: the (input, output) channel counts of the
// network's forward and input-gradient convolutions.
bool launch_brick(const CUtensorMap& tin, const ConvParams& P, int stages, unsigned grid, size_t smem, cudaStream_t s) {
    if (P.cin == 16 && P.cout == 16) launch_brick_t<16, 16>(tin, P, stages, grid, smem, s);
    else if (P.cin == 16 && P.cout == 32) launch_brick_t<16, 32>(tin, P, stages, grid, smem, s);
    else if (P.cin == 32 && P.cout == 16) launch_brick_t<32, 16>(tin, P, stages, grid, smem, s);
    else if (P.cin == 32 && P.cout == 64) launch_brick_t<32, 64>(tin, P, stages, grid, smem, s);
    else if (P.cin == 64 && P.cout == 32) launch_brick_t<64, 32>(tin, P, stages, grid, smem, s);
    else return false;
    return true;
}

void launch_conv(const uint16_t* in, int cin, const uint16_t* w, int cout, const float* bias, int cout_real,
                 const int* d, int mode, const uint16_t* skip, int relu, uint16_t* out_b, float* out_f, NetStatus* st,
                 cudaStream_t s, const int32_t* tiles = nullptr, const int* ntiles_dev = nullptr) {
    ConvParams P;
    P.tiles = nullptr;  // the gathering kernel evaluates every voxel
    P.ntiles = nullptr;
    P.in = in;
    P.cin = cin;
    P.w = w;
    P.cout = cout;
    P.bias = bias;
    P.cout_real = cout_real;
    P.nx = d[0];
    P.ny = d[1];
    P.nz = d[2];
    P.nvox = (long long)d[0] * d[1] * d[2];
    P.mode = mode;
    P.skip = skip;
    P.relu = relu;
    P.out_b = out_b;
    P.out_f = out_f;
    P.status = st;
    if (P.nvox == 0) return;
    // the brick kernel keeps all 27 weight tiles and the brick in shared
    // memory: every layer but the 64 -> 64 input gradient fits
    if (brick_smem_bytes(cin, cout, 1) <= kBrickSmemMax) {
        const int stages = brick_smem_bytes(cin, cout, 2) <= kBrickSmemMax ? 2 : 1;
        const size_t smem = brick_smem_bytes(cin, cout, stages);
        // the input as a 4D tensor (channel, z, y, x), boxes of one 8-channel
        // plane of a brick; zeros outside the grid
        CUtensorMap tin;
        const cuuint64_t dims[4] = {cuuint64_t(cin), cuuint64_t(d[2]), cuuint64_t(d[1]), cuuint64_t(d[0])};
        const cuuint64_t strides[3] = {cuuint64_t(cin) * 2, cuuint64_t(cin) * 2 * d[2],
                                       cuuint64_t(cin) * 2 * d[2] * d[1]};
        const cuuint32_t box[4] = {8, cuuint32_t(kBrZ), cuuint32_t(kBrY), cuuint32_t(kBrX)};
        const cuuint32_t estr[4] = {1, 1, 1, 1};
        const CUresult r = tensor_map_encoder()(&tin, CU_TENSOR_MAP_DATA_TYPE_UINT16, 4, const_cast<uint16_t*>(in),
                                                dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                                CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS)
            throw CudaError(cudaErrorInvalidValue, "brick tensor map: cuTensorMapEncodeTiled failed with CUresult " +
                                                       std::to_string(int(r)));
        const long long ntiles = (long long)d[0] * ((d[1] + 15) / 16) * ((d[2] + 7) / 8);
        const long long per_sm = std::max<long long>(1, (228LL * 1024) / (long long)(smem + 1024));
        const unsigned grid = unsigned(std::min<long long>(ntiles, kSMs * per_sm));
        P.tiles = tiles;
        P.ntiles = tiles ? ntiles_dev : nullptr;
        if (launch_brick(tin, P, stages, grid, smem, s)) return;
        P.tiles = nullptr;  // no instance for these channel counts: the gathering kernel
        P.ntiles = nullptr;
    }
    const size_t smem = size_t(2) * kConvM * cin * 2 + size_t(2) * cout * cin * 2 + 32;
    k_conv<<<unsigned((P.nvox + kConvM - 1) / kConvM), kConvM, smem, s>>>(P);
    LHI_LAUNCH_CHECK();
}

template <int COUT, int CIN> void launch_wgrad_t(WgradParams P, cudaStream_t s) {
    constexpr int smem = WgradTile<COUT, CIN>::kSmem;
    constexpr int groups = (kNetTaps * COUT + 127) / 128;
    LHI_CUDA(cudaFuncSetAttribute(k_wgrad<COUT, CIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    // whole waves of CTAs, of at most kWgChunksPerCta chunks each
    const long long chunks = (P.nvox + kWgChunk - 1) / kWgChunk, slots = kWgCtas * kSMs;
    const long long waves = (chunks * groups + slots * kWgChunksPerCta - 1) / (slots * kWgChunksPerCta);
    P.chunks = int((chunks * groups + slots * waves - 1) / (slots * waves));
    dim3 grid(unsigned((chunks + P.chunks - 1) / P.chunks), groups);
    k_wgrad<COUT, CIN><<<grid, kWgThreads, smem, s>>>(P);
    LHI_LAUNCH_CHECK();
}

void launch_wgrad(const uint16_t* g, int cout, int cout_real, const uint16_t* in, int cin, int cin_real, const int* d,
                  float* grad_w, NetStatus* st, cudaStream_t s) {
    WgradParams P;
    P.g = g;
    P.cout_real = cout_real;
    P.in = in;
    P.cin_real = cin_real;
    P.nx = d[0];
    P.ny = d[1];
    P.nz = d[2];
    P.nvox = (long long)d[0] * d[1] * d[2];
    P.chunks = 0;
    P.grad_w = grad_w;
    P.status = st;
    if (P.nvox == 0) return;
    // the network's (output, input) channel counts
    if (cout == 16 && cin == 16) launch_wgrad_t<16, 16>(P, s);
    else if (cout == 16 && cin == 32) launch_wgrad_t<16, 32>(P, s);
    else if (cout == 32 && cin == 16) launch_wgrad_t<32, 16>(P, s);
    else if (cout == 32 && cin == 64) launch_wgrad_t<32, 64>(P, s);
    else if (cout == 64 && cin == 32) launch_wgrad_t<64, 32>(P, s);
    else throw std::invalid_argument("weight gradient: no instance for these channel counts");
}
}  // namespace

// Needed voxel sets, from the output back to the input (F = type != 0;
// dil = one-voxel dilation; up = coarse voxels with a needed child;
// down = fine voxels with a needed parent):
//   conv5 out F                      (T5)   u0 needed on D = dil(F)
//   conv4 out D (skip h0 on D)       (T4)   q0 needed on dil(D)
//   u1 needed on U1 = up(dil(D))
//   conv3 out U1 (skip h1 on U1)     (T3)   q1 needed on dil(U1)
//   h2 needed on U2 = up(dil(U1))
//   conv2 out U2                     (T2)   p1 needed on dil(U2)
//   h1 needed on H1 = U1 | down(dil(U2))
//   conv1 out H1                     (T1)   p0 needed on dil(H1)
//   h0 needed on H0 = D | down(dil(H1))
//   conv0 out H0                     (T0)   a0 needed on dil(H0): computed everywhere
// Masks: level 0 A, B; level 1 P, Q; level 2 U, W.
void LearnedNet::plan_sparse(const int dims[3], const uint8_t* type, cudaStream_t s) {
    plan_type_ = nullptr;  // no plan until this one is complete
    reserve(dims, true);
    const int* d0 = b_.dims[0];
    const int* d1 = b_.dims[1];
    const int* d2 = b_.dims[2];
    const long long V0 = b_.vox[0];
    size_t m = 0;
    for (auto& p : mask_) p = plan_mem_.at<uint8_t>(m++);
    for (auto& p : tflag_) p = plan_mem_.at<uint8_t>(m++);
    for (auto& p : tlist_) p = plan_mem_.at<int32_t>(m++);
    tcount_ = plan_mem_.at<int>(m);
    uint8_t *A = mask_[0], *B = mask_[1], *P = mask_[2], *Q = mask_[3], *U = mask_[4], *W = mask_[5];
    uint8_t* S = mask_[6];  // the dilations' intermediate (sized for level 0, used at every level)
    LHI_CUDA(cudaMemsetAsync(tcount_, 0, sizeof(int) * kPlanLists, s));
    auto dil = [&](const uint8_t* in, const int* d, uint8_t* out) {
        const long long n = (long long)d[0] * d[1] * d[2];
        if (n == 0) return;
        if (d[2] % 4 == 0) {  // 4-voxel words (the mask buffers are 256-byte aligned)
            const long long nw = n / 4;
            k_mask_dilate4<<<nb(nw), 256, 0, s>>>(reinterpret_cast<const uint32_t*>(in), d[0], d[1], d[2] / 4, 0,
                                                  reinterpret_cast<uint32_t*>(S));
            LHI_LAUNCH_CHECK();
            k_mask_dilate4<<<nb(nw), 256, 0, s>>>(reinterpret_cast<const uint32_t*>(S), d[0], d[1], d[2] / 4, 1,
                                                  reinterpret_cast<uint32_t*>(out));
            LHI_LAUNCH_CHECK();
            return;
        }
        k_mask_dilate<<<nb(n), 256, 0, s>>>(in, d[0], d[1], d[2], 0, S);
        LHI_LAUNCH_CHECK();
        k_mask_dilate<<<nb(n), 256, 0, s>>>(S, d[0], d[1], d[2], 1, out);
        LHI_LAUNCH_CHECK();
    };
    auto up = [&](const uint8_t* fine, const int* fd, const int* cd, uint8_t* coarse) {
        const long long n = (long long)cd[0] * cd[1] * cd[2];
        if (n == 0) return;
        k_mask_up<<<nb(n), 256, 0, s>>>(fine, fd[1], fd[2], cd[0], cd[1], cd[2], coarse);
        LHI_LAUNCH_CHECK();
    };
    auto down_or = [&](const uint8_t* coarse, const int* cd, const uint8_t* other, const int* fd, uint8_t* out) {
        const long long n = (long long)fd[0] * fd[1] * fd[2];
        if (n == 0) return;
        k_mask_down_or<<<nb(n), 256, 0, s>>>(coarse, cd[0], cd[1], cd[2], other, fd[0], fd[1], fd[2], out);
        LHI_LAUNCH_CHECK();
    };
    auto tiles = [&](const uint8_t* m, const int* d, int level, int layer) {
        const long long n = (long long)d[0] * d[1] * d[2], nt = brick_tiles(d);
        if (n == 0) return;
        LHI_CUDA(cudaMemsetAsync(tflag_[level], 0, size_t(nt), s));
        if (d[2] % 4 == 0)
            k_mask_tile_flags4<<<nb(n / 4), 256, 0, s>>>(reinterpret_cast<const uint32_t*>(m), d[0], d[1], d[2] / 4,
                                                         d[2], tflag_[level]);
        else
            k_mask_tile_flags<<<nb(n), 256, 0, s>>>(m, d[0], d[1], d[2], tflag_[level]);
        LHI_LAUNCH_CHECK();
        k_mask_tile_list<<<nb(nt), 256, 0, s>>>(tflag_[level], nt, tlist_[layer], tcount_ + layer);
        LHI_LAUNCH_CHECK();
    };
    k_mask_type<<<nb(V0), 256, 0, s>>>(type, V0, A);  // A = F
    LHI_LAUNCH_CHECK();
    tiles(A, d0, 0, 5);
    dil(A, d0, B);  // B = D
    tiles(B, d0, 0, 4);
    dil(B, d0, A);  // A = dil(D): q0 needed
    tiles(A, d0, 0, kPlanUp0);
    up(A, d0, d1, P);  // P = U1
    tiles(P, d1, 1, 3);
    dil(P, d1, Q);  // q1 needed
    tiles(Q, d1, 1, kPlanUp1);
    up(Q, d1, d2, U);  // U = U2
    tiles(U, d2, 2, 2);
    dil(U, d2, W);  // p1 needed
    tiles(W, d2, 2, kPlanPool1);
    down_or(W, d2, P, d1, Q);  // Q = H1
    tiles(Q, d1, 1, 1);
    dil(Q, d1, P);  // p0 needed
    tiles(P, d1, 1, kPlanPool0);
    down_or(P, d1, B, d0, A);  // A = H0
    tiles(A, d0, 0, 0);
    dil(A, d0, B);  // a0 needed
    tiles(B, d0, 0, kPlanInput);
    plan_type_ = type;
    for (int a = 0; a < 3; ++a) plan_dims_[a] = dims[a];
}

void LearnedNet::forward(const int dims[3], const float* r, const uint8_t* type, const uint8_t* solid, float* z,
                         double scale_fixed, cudaStream_t s, bool sparse) {
    ensure(dims);
    sparse = sparse && sparse_enabled_ && plan_type_ == type && plan_dims_[0] == dims[0] &&
             plan_dims_[1] == dims[1] && plan_dims_[2] == dims[2];
    auto TL = [&](int l) -> const int32_t* { return sparse ? tlist_[l] : nullptr; };
    auto TC = [&](int l) -> const int* { return sparse ? tcount_ + l : nullptr; };
    if (wfmt_stale_) format_weights(s);
    last_type_ = type;
    const int* d0 = b_.dims[0];
    const int* d1 = b_.dims[1];
    const int* d2 = b_.dims[2];
    const long long V0 = b_.vox[0];
    if (scale_fixed > 0) {
        const float sf = float(scale_fixed);
        LHI_CUDA(cudaMemcpyAsync(scale_, &sf, sizeof(float), cudaMemcpyHostToDevice, s));
    } else {
        k_net_scale<<<std::min<unsigned>(nb(V0), 1024), 256, 0, s>>>(r, type, V0, red_, counter_, scale_);
        LHI_LAUNCH_CHECK();
    }
    // the elementwise stages on their plan's tiles: a persistent grid
    const auto tgrid = [](const int* d) {
        return unsigned(std::max(1LL, std::min<long long>(brick_tiles(d), (long long)kSMs * 16)));
    };
    if (sparse)
        k_net_input_tiles<<<tgrid(d0), 128, 0, s>>>(r, type, solid, d0[0], d0[1], d0[2], scale_, b_.a0,
                                                    tlist_[kPlanInput], tcount_ + kPlanInput);
    else
        k_net_input<<<nb(V0), 256, 0, s>>>(r, type, solid, d0[0], d0[1], d0[2], scale_, b_.a0);
    LHI_LAUNCH_CHECK();
    auto W = [&](int l) { return wfwd_ + wfwd_off_[l]; };
    // bias-free: M(0) = 0 (the packed bias entries are kept and ignored)
    auto Bv = [&](int l) -> const float* {
        (void)l;
        return nullptr;
    };
    const int act = relu_ ? 1 : 0;
    launch_conv(b_.a0, 16, W(0), 16, Bv(0), 16, d0, 0, nullptr, act, b_.h0, nullptr, status_, s, TL(0), TC(0));
    if (sparse)
        k_pool_tiles<<<tgrid(d1), 128, 0, s>>>(b_.h0, d0[1], d0[2], b_.p0, d1[1], d1[2], 16, tlist_[kPlanPool0],
                                               tcount_ + kPlanPool0);
    else
        k_pool<<<nb(b_.vox[1] * 16 / 8), 256, 0, s>>>(b_.h0, d0[1], d0[2], b_.p0, d1[0], d1[1], d1[2], 16);
    LHI_LAUNCH_CHECK();
    launch_conv(b_.p0, 16, W(1), 32, Bv(1), 32, d1, 0, nullptr, act, b_.h1, nullptr, status_, s, TL(1), TC(1));
    if (sparse)
        k_pool_tiles<<<tgrid(d2), 128, 0, s>>>(b_.h1, d1[1], d1[2], b_.p1, d2[1], d2[2], 32, tlist_[kPlanPool1],
                                               tcount_ + kPlanPool1);
    else
        k_pool<<<nb(b_.vox[2] * 32 / 8), 256, 0, s>>>(b_.h1, d1[1], d1[2], b_.p1, d2[0], d2[1], d2[2], 32);
    LHI_LAUNCH_CHECK();
    launch_conv(b_.p1, 32, W(2), 64, Bv(2), 64, d2, 0, nullptr, act, b_.h2, nullptr, status_, s, TL(2), TC(2));
    if (sparse)
        k_upsample_tiles<<<tgrid(d1), 128, 0, s>>>(b_.h2, d2[0], d2[1], d2[2], b_.q1, d1[1], d1[2], 64,
                                                   tlist_[kPlanUp1], tcount_ + kPlanUp1);
    else
        k_upsample<<<nb(b_.vox[1] * 64 / 8), 256, 0, s>>>(b_.h2, d2[0], d2[1], d2[2], b_.q1, d1[0], d1[1], d1[2], 64);
    LHI_LAUNCH_CHECK();
    launch_conv(b_.q1, 64, W(3), 32, Bv(3), 32, d1, 0, b_.h1, act, b_.u1, nullptr, status_, s, TL(3), TC(3));
    if (sparse)
        k_upsample_tiles<<<tgrid(d0), 128, 0, s>>>(b_.u1, d1[0], d1[1], d1[2], b_.q0, d0[1], d0[2], 32,
                                                   tlist_[kPlanUp0], tcount_ + kPlanUp0);
    else
        k_upsample<<<nb(V0 * 32 / 8), 256, 0, s>>>(b_.u1, d1[0], d1[1], d1[2], b_.q0, d0[0], d0[1], d0[2], 32);
    LHI_LAUNCH_CHECK();
    launch_conv(b_.q0, 32, W(4), 16, Bv(4), 16, d0, 0, b_.h0, act, b_.u0, nullptr, status_, s, TL(4), TC(4));
    launch_conv(b_.u0, 16, W(5), 16, Bv(5), 1, d0, 2, nullptr, 0, nullptr, b_.y, status_, s, TL(5), TC(5));
    k_net_output<<<nb(V0), 256, 0, s>>>(b_.y, type, V0, scale_, z);
    LHI_LAUNCH_CHECK();
}

void LearnedNet::backward(const float* dz, cudaStream_t s) {
    const int* d0 = b_.dims[0];
    const int* d1 = b_.dims[1];
    const int* d2 = b_.dims[2];
    const long long V0 = b_.vox[0], V1 = b_.vox[1], V2 = b_.vox[2];
    auto WB = [&](int l) { return wbwd_ + wbwd_off_[l]; };
    auto GW = [&](int l) { return grad_ + net_param_offset(l); };
    // the network is bias-free: the packed bias entries keep zero gradient
    // layer 5
    k_net_dy<<<nb(V0), 256, 0, s>>>(dz, last_type_, V0, scale_, b_.g[5]);
    LHI_LAUNCH_CHECK();
    launch_wgrad(b_.g[5], 16, 1, b_.u0, 16, 16, d0, GW(5), status_, s);
    launch_conv(b_.g[5], 16, WB(5), 16, nullptr, 16, d0, 1, nullptr, 0, nullptr, b_.dx, status_, s);
    // layer 4
    k_relu_grad<<<nb(V0 * 16 / 8), 256, 0, s>>>(b_.dx, b_.u0, V0 * 16 / 8, relu_ ? 1 : 0, b_.g[4]);
    LHI_LAUNCH_CHECK();
    launch_wgrad(b_.g[4], 16, 16, b_.q0, 32, 32, d0, GW(4), status_, s);
    launch_conv(b_.g[4], 16, WB(4), 32, nullptr, 32, d0, 1, nullptr, 0, nullptr, b_.dx, status_, s);
    k_sum_children<<<nb(V1 * 32 / 8), 256, 0, s>>>(b_.dx, d0[1], d0[2], b_.acc, d1[0], d1[1], d1[2], 32);
    LHI_LAUNCH_CHECK();
    // layer 3
    k_relu_grad<<<nb(V1 * 32 / 8), 256, 0, s>>>(b_.acc, b_.u1, V1 * 32 / 8, relu_ ? 1 : 0, b_.g[3]);
    LHI_LAUNCH_CHECK();
    launch_wgrad(b_.g[3], 32, 32, b_.q1, 64, 64, d1, GW(3), status_, s);
    launch_conv(b_.g[3], 32, WB(3), 64, nullptr, 64, d1, 1, nullptr, 0, nullptr, b_.dx, status_, s);
    k_sum_children<<<nb(V2 * 64 / 8), 256, 0, s>>>(b_.dx, d1[1], d1[2], b_.acc, d2[0], d2[1], d2[2], 64);
    LHI_LAUNCH_CHECK();
    // layer 2
    k_relu_grad<<<nb(V2 * 64 / 8), 256, 0, s>>>(b_.acc, b_.h2, V2 * 64 / 8, relu_ ? 1 : 0, b_.g[2]);
    LHI_LAUNCH_CHECK();
    launch_wgrad(b_.g[2], 64, 64, b_.p1, 32, 32, d2, GW(2), status_, s);
    launch_conv(b_.g[2], 64, WB(2), 32, nullptr, 32, d2, 1, nullptr, 0, nullptr, b_.dx, status_, s);
    // layer 1: dh1 = g3 (skip) + unpool(dp1) / 8
    k_relu_grad_unpool<<<nb(V1 * 32 / 8), 256, 0, s>>>(b_.g[3], b_.dx, d2[0], d2[1], d2[2], b_.h1, d1[0], d1[1], d1[2],
                                                       32, relu_ ? 1 : 0, b_.g[1]);
    LHI_LAUNCH_CHECK();
    launch_wgrad(b_.g[1], 32, 32, b_.p0, 16, 16, d1, GW(1), status_, s);
    launch_conv(b_.g[1], 32, WB(1), 16, nullptr, 16, d1, 1, nullptr, 0, nullptr, b_.dx, status_, s);
    // layer 0: dh0 = g4 (skip) + unpool(dp0) / 8
    k_relu_grad_unpool<<<nb(V0 * 16 / 8), 256, 0, s>>>(b_.g[4], b_.dx, d1[0], d1[1], d1[2], b_.h0, d0[0], d0[1], d0[2],
                                                       16, relu_ ? 1 : 0, b_.g[0]);
    LHI_LAUNCH_CHECK();
    launch_wgrad(b_.g[0], 16, 16, b_.a0, 16, 4, d0, GW(0), status_, s);
}

int umma_selftest(const uint16_t* a_host, const uint16_t* b_host, int N, int K, float* d_host, int* stage) {
    if (N < 16 || N > 64 || N % 16 || K < 16 || K > 64 || K % 16) throw std::invalid_argument("selftest: N, K in {16, 32, 48, 64}");
    uint16_t *a = nullptr, *b = nullptr;
    float* d = nullptr;
    NetStatus* st = nullptr;
    LHI_CUDA(cudaMalloc(&a, 2 * 128 * K));
    LHI_CUDA(cudaMalloc(&b, 2 * N * K));
    LHI_CUDA(cudaMalloc(&d, 4 * 128 * N));
    LHI_CUDA(cudaMalloc(&st, sizeof(NetStatus)));
    LHI_CUDA(cudaMemset(st, 0, sizeof(NetStatus)));
    LHI_CUDA(cudaMemset(d, 0, 4 * 128 * N));
    LHI_CUDA(cudaMemcpy(a, a_host, 2 * 128 * K, cudaMemcpyHostToDevice));
    LHI_CUDA(cudaMemcpy(b, b_host, 2 * N * K, cudaMemcpyHostToDevice));
    k_umma_selftest<<<1, 128>>>(a, b, N, K, d, st);
    LHI_LAUNCH_CHECK();
    LHI_CUDA(cudaDeviceSynchronize());
    NetStatus h{};
    LHI_CUDA(cudaMemcpy(&h, st, sizeof(h), cudaMemcpyDeviceToHost));
    LHI_CUDA(cudaMemcpy(d_host, d, 4 * 128 * N, cudaMemcpyDeviceToHost));
    cudaFree(a);
    cudaFree(b);
    cudaFree(d);
    cudaFree(st);
    *stage = h.pad[3];
    return h.timeout ? LHI_E_TIMEOUT : LHI_OK;
}

void LearnedNet::adam_step(double lr, double beta1, double beta2, double eps, cudaStream_t s) {
    ++adam_t_;
    const double c1 = 1.0 - std::pow(beta1, double(adam_t_));
    const double c2 = 1.0 - std::pow(beta2, double(adam_t_));
    const long long n = net_param_count();
    k_adam<<<nb(n), 256, 0, s>>>(w32_, grad_, adam_m_, adam_v_, n, float(lr), float(beta1), float(beta2), float(eps),
                                 float(c1), float(c2));
    LHI_LAUNCH_CHECK();
    wfmt_stale_ = true;
}

}  // namespace lhi
