// el_nn.cu -- the learned warm start's network kernels: BF16 implicit-GEMM 3x3x3 convolutions
// on the tensor cores (mma.sync m16n8k16, FP32 accumulation), forward and both backward passes,
// and the small kernels around them (pooling, upsampling, the 1x1x1 head with its loss, Adam,
// weight packing).  No counterpart in the reference, which has no learned component.
//
// Layout: activations are channels-last bf16, element (x, y, z, c) at ((z*Y + y)*X + x)*C + c,
// one sample per call.  A convolution's input may be the concatenation of two tensors (the
// decoder's [upsampled coarse, skip]) with the upsampling (nearest, factor 2) folded into the
// load: nothing concatenated or upsampled is ever written out.
//
// Forward = implicit GEMM with M = output voxels, N = output channels, K = 27 taps x input
// channels.  A CTA owns a 16 (x) x 8 (y) x 1 (z) brick of output voxels, one warp per y row:
// the input brick with its one-voxel halo (18 x 10 x 3 voxels, all input channels) is staged
// once in shared memory and the 27 taps read it through ldmatrix at shifted rows.  Weights are
// pre-packed in the mma B-fragment order, so each lane fetches its fragments with one 16-byte
// load per pair of n-blocks (they stay in L1: every warp of the CTA reads the same ones).
//
// Backward data is the same kernel: grad_in = conv(grad_out masked by ReLU', W') with W' the
// weights transposed in channels and mirrored in taps (packed separately); its output splits
// back into the two concatenated inputs.  Backward weight is a second implicit GEMM,
// M = output channels, N = input channels, K = voxels, per tap; a CTA takes all 27 taps of 16 input
// channels over a range of planes, accumulators in registers, and writes one partial, summed in a
// fixed order by a reduction kernel (deterministic).
#include <cuda_bf16.h>

#include <cstdint>

#include "el_internal.cuh"

namespace el {
namespace nn {

constexpr int kTX = 16, kTY = 8;                     // output brick (x, y); z = 1
constexpr int kHX = kTX + 2, kHY = kTY + 2, kHZ = 3;  // with halo
constexpr int kHV = kHX * kHY * kHZ;                 // 540 halo voxels
constexpr int kThreads = 256;

struct ConvIn {
    const __nv_bfloat16* a;  // channels [0, ca)
    const __nv_bfloat16* b;  // channels [ca, ca + cb), fine resolution; NULL: cb channels of zeros
    const __nv_bfloat16* mask;  // optional, fine resolution, ca + cb channels: zero where <= 0
    int ca, cb, up_a;           // up_a: `a` is at half resolution (nearest upsampling)
    int ax, ay, az;             // dims of `a`
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// 16 bytes to shared memory, zeros where !valid (src is then any valid address)
__device__ __forceinline__ void cp_async16_zfill(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}

__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// zero the bf16 lanes of v whose mask lane is not > 0 (bf16 sign/magnitude test)
__device__ __forceinline__ uint4 apply_relu_mask(uint4 v, uint4 m) {
    uint32_t* pv = reinterpret_cast<uint32_t*>(&v);
    const uint32_t* pm = reinterpret_cast<const uint32_t*>(&m);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uint32_t keep = 0;
        const uint32_t lo = pm[q] & 0xffffu, hi = pm[q] >> 16;
        // > 0: sign bit clear and not +0
        if (!(lo & 0x8000u) && lo != 0u) keep |= 0x0000ffffu;
        if (!(hi & 0x8000u) && hi != 0u) keep |= 0xffff0000u;
        pv[q] &= keep;
    }
    return v;
}

// Stage the input brick (with halo) of output brick (x0, y0, z0) into smem rows of `srow`
// bf16 (channel-contiguous, 16 bytes of padding per row against bank conflicts).
template <int CIN>
__device__ __forceinline__ void stage_halo(__nv_bfloat16* halo, const ConvIn& in, int X, int Y, int Z, int x0, int y0,
                                           int z0) {
    constexpr int CV = CIN / 8;
    constexpr int SROW = CIN + 8;
    for (int idx = threadIdx.x; idx < kHV * CV; idx += kThreads) {
        const int hv = idx / CV, cv = idx - hv * CV;
        const int hx = hv % kHX, t = hv / kHX, hy = t % kHY, hz = t / kHY;
        const int x = x0 + hx - 1, y = y0 + hy - 1, z = z0 + hz - 1;
        uint4 val = make_uint4(0u, 0u, 0u, 0u);
        if (x >= 0 && x < X && y >= 0 && y < Y && z >= 0 && z < Z) {
            const int c = cv * 8;
            const long long fine = ((long long)z * Y + y) * X + x;
            if (c < in.ca) {
                const long long va = in.up_a ? ((long long)(z >> 1) * in.ay + (y >> 1)) * in.ax + (x >> 1) : fine;
                val = __ldg(reinterpret_cast<const uint4*>(in.a + va * in.ca + c));
            } else if (in.b) {
                val = __ldg(reinterpret_cast<const uint4*>(in.b + fine * in.cb + (c - in.ca)));
            }
            if (in.mask) val = apply_relu_mask(val, __ldg(reinterpret_cast<const uint4*>(in.mask + fine * CIN + c)));
        }
        *reinterpret_cast<uint4*>(halo + hv * SROW + cv * 8) = val;
    }
}

// ---------------------------------------------------------------------------------------
// forward / backward-data convolution
template <int CIN, int COUT>
__global__ void __launch_bounds__(kThreads) conv3_kernel(int X, int Y, int Z, ConvIn in, const uint4* __restrict__ wf,
                                                         const float* __restrict__ bias, int relu,
                                                         __nv_bfloat16* __restrict__ out_a, int oca,
                                                         __nv_bfloat16* __restrict__ out_b) {
    constexpr int KS = CIN / 16, NB = COUT / 8, SROW = CIN + 8;
    static_assert(CIN % 16 == 0 && COUT % 16 == 0, "channels must be multiples of 16");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __nv_bfloat16* halo = reinterpret_cast<__nv_bfloat16*>(smem_raw);
    const int x0 = blockIdx.x * kTX, y0 = blockIdx.y * kTY, z0 = blockIdx.z;
    stage_halo<CIN>(halo, in, X, Y, Z, x0, y0, z0);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float acc[NB][4];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) acc[nb][0] = acc[nb][1] = acc[nb][2] = acc[nb][3] = 0.f;
    // ldmatrix row of this lane: voxel x = r, channel offset kofs within the 16-channel step
    const int r = (lane & 7) + ((lane >> 3) & 1) * 8, kofs = (lane >> 4) * 8;
#pragma unroll 1
    for (int tap = 0; tap < 27; ++tap) {
        const int dz = tap / 9 - 1, dy = (tap / 3) % 3 - 1, dx = tap % 3 - 1;
        const int hv = ((1 + dz) * kHY + (warp + 1 + dy)) * kHX + (1 + dx) + r;
        const uint32_t abase = smem_u32(halo + hv * SROW + kofs);
        const uint4* wp = wf + (size_t)tap * KS * (NB / 2) * 32 + lane;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
            uint32_t a[4];
            ldsm_x4(abase + ks * 32, a);
#pragma unroll
            for (int p = 0; p < NB / 2; ++p) {
                const uint4 b = __ldg(wp + (ks * (NB / 2) + p) * 32);
                mma_bf16(acc[2 * p], a, b.x, b.y);
                mma_bf16(acc[2 * p + 1], a, b.z, b.w);
            }
        }
    }
    const int y = y0 + warp;
    if (y >= Y) return;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int x = x0 + (lane >> 2) + 8 * h;
        if (x >= X) continue;
        const long long v = ((long long)z0 * Y + y) * X + x;
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
            const int co = nb * 8 + (lane & 3) * 2;
            float v0 = acc[nb][2 * h], v1 = acc[nb][2 * h + 1];
            if (bias) {
                v0 += bias[co];
                v1 += bias[co + 1];
            }
            if (relu) {
                v0 = fmaxf(v0, 0.f);
                v1 = fmaxf(v1, 0.f);
            }
            const __nv_bfloat162 pr = __floats2bfloat162_rn(v0, v1);
            if (co < oca)
                *reinterpret_cast<__nv_bfloat162*>(out_a + v * oca + co) = pr;
            else
                *reinterpret_cast<__nv_bfloat162*>(out_b + v * (COUT - oca) + (co - oca)) = pr;
        }
    }
}

// ---------------------------------------------------------------------------------------
// The same convolution on the 5th-generation tensor cores (tcgen05).  A unit is the 8 (x) x 16 (y)
// voxels of one column in one plane z: M = 128 voxels, one TMEM lane each; N = output channels in TMEM
// columns (FP32).  A CTA owns a range of units (z fastest) and takes it in runs within a column, with
// one accumulator per unit of a run; the input channels go in slices of SC.  For each slice it fetches
// the slice's 27 taps of weights (once for all runs, if there is one slice) and marches the run's
// planes; after the last slice the run is stored.  Both operands sit in shared memory in the no-swizzle
// K-major layout, whose unit is an 8-row x 16-byte core matrix:
//   A: a ring of five input planes with their halo (10 x 18 voxels), channel-chunk major: chunk c
//      (channels 8c..8c+7) of voxel v of ring slot s at ((5 c + s) * 180 + v) * 16 bytes.  Eight
//      x-consecutive voxels are one core matrix, the next 8 rows (the next y) are 10 voxels further
//      (SBO = 160 B), the next chunk along K is five planes further (LBO = 14400 B); tap
//      (dx, dy, dz) only moves the start address, so the 27 shifted operands need no copies.
//   B: per tap, [channel chunk][output channel] x 16 bytes: SBO = 128 B, LBO = cout * 16 B.
// One thread issues the 27 * SC / 16 MMAs (K = 16 each) of a unit and commits them to one of two
// mbarriers; while they run, the plane two units ahead is fetched (cp.async, zero-filled outside the
// grid; with a ReLU mask, through registers).
// A plane of a column is staged once a slice (bricks of one plane staged three, and that staging was
// most of the time), and several CTAs on an SM cover each other's staging: SC and the CTAs an SM are
// chosen together so that weights and ring fit (EL_NN_TC_PAIRS; all 48 channels of 48 -> 16 at once
// left one CTA an SM: 589 us against 222).  An MMA reads 4 KB of A whatever N is, about 32 clocks: that
// and the staging bound the narrow layers (16 -> 16 at 128^3: 48 us of MMA).  Forward / backward data,
// before (bricks) and now: 16 -> 16 at 128^3 166 / 258 -> 88 / 116 us; 32 -> 96 at 64^3 196 -> 66.
namespace tc {

__device__ int g_error;  // set when a bounded wait gave up; read and cleared by el_nn_take_error

constexpr int TX = 8, TY = 16, HX = TX + 2, HY = TY + 2, PV = HX * HY;  // 180 voxels of a staged plane
constexpr int kThreads = 256;
constexpr int kRing = 5;     // planes z - 1, z, z + 1 of a unit, z + 2 landing, z + 3 on its way

__device__ __forceinline__ int ring_slot(int z) { return (int)((unsigned)(z + kRing) % (unsigned)kRing); }

template <int CIN, int COUT>
struct Shape {
    static constexpr int KC = CIN / 8;                 // 16-byte channel chunks
    static constexpr int WB = 27 * KC * COUT * 16;     // weight bytes
    static constexpr int LBO = kRing * PV * 16;            // bytes from a channel chunk to the next
    static constexpr int HB = KC * LBO;                // the ring
    static constexpr int SMEM = WB + HB + COUT * 4 + 32;  // + bias, two mbarriers and the TMEM address
    // BF16 x BF16 -> FP32, both K-major, M = 128, N = COUT
    static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(COUT >> 3) << 17) |
                                      ((uint32_t)(128 >> 4) << 24);
};

__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo & 0x3FFFFu) >> 4) << 16;
    d |= (uint64_t)((sbo & 0x3FFFFu) >> 4) << 32;
    d |= (uint64_t)1 << 46;  // descriptor version of the 5th-generation tensor cores; no swizzle
    return d;
}

__device__ __forceinline__ bool mbar_wait(uint32_t addr, uint32_t phase) {
    // polls without suspending; gives up (and reports) after about two seconds of SM clock
    const long long start = clock64();
    while (true) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(addr), "r"(phase)
            : "memory");
        if (done) return true;
        if (clock64() - start > (1LL << 32)) return false;
    }
}

// The staging of a column's planes, KC channel chunks from chunk c0 of the input on.  Chunk idx of a
// plane: voxel idx / KC, channel chunk idx % KC (consecutive threads read consecutive bytes of a
// voxel); a thread's chunks are the same in every plane, so what depends on x and y is formed once a
// column.
template <int KC>
struct ColumnStage {
    static constexpr int N = PV * KC, PER = (N + kThreads - 1) / kThreads;
    int va[PER], vf[PER];  // voxel within a plane of `a`, and at full resolution (-1: outside the grid)
    __device__ __forceinline__ void column(const ConvIn& in, int X, int Y, int x0, int y0) {
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const int hv = ((int)threadIdx.x + q * kThreads) / KC, hy = hv / HX, hx = hv - hy * HX;
            const int x = x0 + hx - 1, y = y0 + hy - 1;
            const bool inside = hv < PV && x >= 0 && x < X && y >= 0 && y < Y;
            vf[q] = inside ? y * X + x : -1;
            va[q] = in.up_a ? (y >> 1) * in.ax + (x >> 1) : vf[q];
        }
    }
    // plane z into its ring slot
    __device__ __forceinline__ void plane(unsigned char* ring, const ConvIn& in, int X, int Y, int Z, int c0, int z) const {
        constexpr int LBO = kRing * PV * 16;
        unsigned char* slot = ring + (size_t)ring_slot(z) * PV * 16;
        const bool z_in = z >= 0 && z < Z;
        const long long pa = (long long)(in.up_a ? z >> 1 : z) * in.ax * in.ay, pf = (long long)z * X * Y;
        auto source = [&](int q) -> const __nv_bfloat16* {
            const int c = (c0 + ((int)threadIdx.x + q * kThreads) % KC) * 8;
            if (!z_in || vf[q] < 0) return nullptr;
            if (c < in.ca) return in.a + (pa + va[q]) * in.ca + c;
            return in.b ? in.b + (pf + vf[q]) * in.cb + (c - in.ca) : nullptr;
        };
        if (in.mask) {  // the mask is applied on the way: through registers, a few chunks in flight
            constexpr int U = PER < 3 ? PER : 3;
#pragma unroll
            for (int q0 = 0; q0 < PER; q0 += U) {
                uint4 v[U], m[U];
#pragma unroll
                for (int q = 0; q < U; ++q) {
                    const __nv_bfloat16* p = q0 + q < PER ? source(q0 + q) : nullptr;
                    const int c = (c0 + ((int)threadIdx.x + (q0 + q) * kThreads) % KC) * 8;
                    v[q] = m[q] = make_uint4(0u, 0u, 0u, 0u);
                    if (p) {
                        v[q] = __ldg(reinterpret_cast<const uint4*>(p));
                        m[q] = __ldg(reinterpret_cast<const uint4*>(in.mask + (pf + vf[q0 + q]) * (in.ca + in.cb) + c));
                    }
                }
#pragma unroll
                for (int q = 0; q < U; ++q) {
                    const int idx = (int)threadIdx.x + (q0 + q) * kThreads;
                    if (q0 + q < PER && idx < N)
                        *reinterpret_cast<uint4*>(slot + (size_t)(idx % KC) * LBO + (idx / KC) * 16) =
                            apply_relu_mask(v[q], m[q]);
                }
            }
            return;
        }
        const uint32_t base = smem_u32(slot);
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const int idx = (int)threadIdx.x + q * kThreads;
            if (idx >= N) break;
            const __nv_bfloat16* p = source(q);
            cp_async16_zfill(base + (uint32_t)((idx % KC) * LBO + (idx / KC) * 16), p ? p : in.a, p != nullptr);
        }
    }
};

// accumulator columns [col, col + COUT) of this warp's 32 lanes -> bias, ReLU, bf16, store; the two
// warps of a lane quarter take alternate groups of 16 channels (bias: in shared memory)
template <int COUT>
__device__ __forceinline__ void tc_epilogue(uint32_t tmem, uint32_t col, int X, int Y, int x0, int y0, int z0,
                                            const float* bias, int relu, __nv_bfloat16* out_a, int oca,
                                            __nv_bfloat16* out_b) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int x = x0 + (r & 7), y = y0 + (r >> 3);
    const bool live = x < X && y < Y;
    const long long v = ((long long)z0 * Y + y) * X + x;
#pragma unroll
    for (int c0 = 0; c0 < COUT; c0 += 16) {
        if (((c0 >> 4) & 1) != (warp >> 2)) continue;
        uint32_t q[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
            "[%16];\n"
            : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]), "=r"(q[4]), "=r"(q[5]), "=r"(q[6]), "=r"(q[7]),
              "=r"(q[8]), "=r"(q[9]), "=r"(q[10]), "=r"(q[11]), "=r"(q[12]), "=r"(q[13]), "=r"(q[14]), "=r"(q[15])
            : "r"(tmem + ((uint32_t)(quarter * 32) << 16) + col + (uint32_t)c0));
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        if (!live) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint4 o;
            __nv_bfloat162* op = reinterpret_cast<__nv_bfloat162*>(&o);
            const float4 b0 = *reinterpret_cast<const float4*>(bias + c0 + h * 8);
            const float4 b1 = *reinterpret_cast<const float4*>(bias + c0 + h * 8 + 4);
            const float bb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float f0 = __uint_as_float(q[h * 8 + 2 * e]) + bb[2 * e];
                float f1 = __uint_as_float(q[h * 8 + 2 * e + 1]) + bb[2 * e + 1];
                f0 = relu ? fmaxf(f0, 0.f) : f0;
                f1 = relu ? fmaxf(f1, 0.f) : f1;
                op[e] = __floats2bfloat162_rn(f0, f1);
            }
            const int cb = c0 + h * 8;
            if (cb < oca)
                *reinterpret_cast<uint4*>(out_a + v * oca + cb) = o;
            else
                *reinterpret_cast<uint4*>(out_b + v * (COUT - oca) + (cb - oca)) = o;
        }
    }
}

// the MMAs of the unit in plane z into the accumulator at tmem_acc (first: which they start), committed
// to mbar (one thread).  A descriptor's address field counts 16 bytes, so a tap is one addition to it.
template <int CIN, int COUT>
__device__ __forceinline__ void tc_issue(uint32_t tmem_acc, uint32_t ring, uint32_t wbase, uint32_t mbar, int z,
                                         bool first) {
    using S = Shape<CIN, COUT>;
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint64_t d0 = smem_desc(ring, S::LBO, HX * 16);
    uint64_t db = smem_desc(wbase, COUT * 16, 128);
#pragma unroll 1
    for (int dz = 0; dz < 3; ++dz) {
        const uint64_t dplane = d0 + (uint64_t)(ring_slot(z - 1 + dz) * PV);
#pragma unroll
        for (int t = 0; t < 9; ++t)
#pragma unroll
            for (int s = 0; s < S::KC / 2; ++s) {
                const uint64_t da = dplane + (uint64_t)((t / 3) * HX + t % 3 + 2 * s * (S::LBO / 16));
                const uint32_t acc = (!first || (dz | t | s)) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_acc),
                    "l"(da), "l"(db), "r"(S::IDESC), "r"(acc)
                    : "memory");
                db += 2 * COUT;
            }
    }
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(mbar)
                 : "memory");
}

template <int CIN, int COUT, int SC, int CTAS>
struct RunShape {
    using S = Shape<SC, COUT>;                                                      // a slice's layout
    static constexpr int SLICES = CIN / SC;
    static constexpr uint32_t NCOL = CTAS == 1 ? 512u : (CTAS == 2 ? 256u : 128u);  // of the SM's 512
    static constexpr int MAX_RUN = (int)NCOL / COUT < 16 ? (int)NCOL / COUT : 16;   // accumulators
};

template <int CIN, int COUT, int SC, int CTAS>
__global__ void __launch_bounds__(kThreads, CTAS) conv3_tc_kernel(int X, int Y, int Z, ConvIn in,
                                                                      const uint4* __restrict__ wtc,
                                                                      const float* __restrict__ bias, int relu,
                                                                      __nv_bfloat16* __restrict__ out_a, int oca,
                                                                      __nv_bfloat16* __restrict__ out_b) {
    using SS = RunShape<CIN, COUT, SC, CTAS>;
    using S = typename SS::S;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* wsm = smem_raw;
    unsigned char* ring = smem_raw + S::WB;
    float* sbias = reinterpret_cast<float*>(smem_raw + S::WB + S::HB);
    uint64_t* mbar = reinterpret_cast<uint64_t*>(smem_raw + S::WB + S::HB + COUT * 4);  // two
    uint32_t* tslot = reinterpret_cast<uint32_t*>(smem_raw + S::WB + S::HB + COUT * 4 + 16);
    const int tid = threadIdx.x, warp = tid >> 5;
    if (tid < COUT) sbias[tid] = bias ? bias[tid] : 0.f;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tslot)),
                     "r"(SS::NCOL)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(mbar)), "r"(1) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(mbar + 1)), "r"(1) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *tslot;
    const uint32_t wbase = smem_u32(wsm), rbase = smem_u32(ring);
    const uint32_t mb[2] = {smem_u32(mbar), smem_u32(mbar + 1)};
    const int bx = (X + TX - 1) / TX, by = (Y + TY - 1) / TY, per = SS::MAX_RUN;
    const long long units = (long long)bx * by * Z;
    const long long u_end = units * (blockIdx.x + 1) / gridDim.x;
    uint32_t phase[2] = {0u, 0u};
    bool ok = true;
    auto finish_wait = [&](int b) {  // the MMAs committed to mbarrier b; uniform over the block
        const bool mine_ok = mbar_wait(mb[b], phase[b]);
        phase[b] ^= 1u;
        const bool all = __syncthreads_and(mine_ok) != 0;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        return all;
    };
    ColumnStage<S::KC> stage;
    int b = 0;
    bool fresh = true;  // no weights fetched yet
    for (long long u = units * blockIdx.x / gridDim.x; u < u_end && ok;) {
        // what is left of this CTA's units in this column, as runs of about one length
        const long long colu = u / Z;
        const int x0 = (int)(colu % bx) * TX, y0 = (int)(colu / bx) * TY;
        const int z_begin = (int)(u - colu * Z), left = (int)min((long long)(Z - z_begin), u_end - u);
        const int nruns = (left + per - 1) / per, z_end = z_begin + (left + nruns - 1) / nruns;
        u += z_end - z_begin;
        stage.column(in, X, Y, x0, y0);
#pragma unroll 1
        for (int sl = 0; sl < SS::SLICES && ok; ++sl) {
            // every MMA of the slice before has completed: its weights and planes may be overwritten
            const int c0 = sl * S::KC;
            for (int q = tid; q < S::WB / 16 && (SS::SLICES > 1 || fresh); q += kThreads) {
                constexpr int T = S::KC * COUT;  // 16-byte pieces of a tap of the slice
                const int tap = q / T, o = q - tap * T;
                cp_async16_zfill(wbase + (uint32_t)q * 16, wtc + (size_t)tap * (CIN / 8) * COUT + (size_t)c0 * COUT + o, true);
            }
            stage.plane(ring, in, X, Y, Z, c0, z_begin - 1);
            stage.plane(ring, in, X, Y, Z, c0, z_begin);
            stage.plane(ring, in, X, Y, Z, c0, z_begin + 1);
            asm volatile("cp.async.commit_group;\n" ::: "memory");
            if (z_begin + 1 < z_end) stage.plane(ring, in, X, Y, Z, c0, z_begin + 2);
            asm volatile("cp.async.commit_group;\n" ::: "memory");
#pragma unroll 1
            for (int z = z_begin; z < z_end; ++z) {
                asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // plane z + 1 has landed
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                __syncthreads();
                if (tid == 0)
                    tc_issue<SC, COUT>(tmem + (uint32_t)((z - z_begin) * COUT), rbase, wbase, mb[b], z, sl == 0);
                if (z > z_begin) {
                    ok = finish_wait(b ^ 1);  // the slot of plane z - 2 is free
                    if (!ok) break;
                }
                if (z + 2 < z_end) stage.plane(ring, in, X, Y, Z, c0, z + 3);
                asm volatile("cp.async.commit_group;\n" ::: "memory");
                b ^= 1;
            }
            if (ok) ok = finish_wait(b ^ 1);
        }
        if (!ok) break;
        fresh = false;
        for (int z = z_begin; z < z_end; ++z)
            tc_epilogue<COUT>(tmem, (uint32_t)((z - z_begin) * COUT), X, Y, x0, y0, z, sbias, relu, out_a, oca, out_b);
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncthreads();  // the accumulators are read before the next run writes them
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    }
    if (!ok && tid == 0) {
        atomicExch(&g_error, 1);
        mbar_wait(mb[0], phase[0]);  // once more (bounded), for MMAs still in flight
        mbar_wait(mb[1], phase[1]);
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(SS::NCOL) : "memory");
}

// FP32 master [co][27][ci] -> the B layout above: [tap][ci / 8][co][ci % 8]
__global__ void pack_weights_tc_kernel(int cin, int cout, const float* __restrict__ w, __nv_bfloat16* __restrict__ tf,
                                       __nv_bfloat16* __restrict__ tb) {
    const long long n = 27LL * cin * cout;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const int ci = (int)(e % cin);
        const long long t2 = e / cin;
        const int tap = (int)(t2 % 27), co = (int)(t2 / 27);
        const __nv_bfloat16 v = __float2bfloat16_rn(w[e]);
        tf[(((size_t)tap * (cin / 8) + ci / 8) * cout + co) * 8 + (ci % 8)] = v;
        // backward data: the transposed, tap-mirrored kernel (cin' = cout, cout' = cin)
        if (tb) tb[(((size_t)(26 - tap) * (cout / 8) + co / 8) * cin + ci) * 8 + (co % 8)] = v;
    }
}

}  // namespace tc

// ---------------------------------------------------------------------------------------
// backward weight: dW[co][tap][ci] = sum_v gm[v][co] x[v + off(tap)][ci], gm = g * (y > 0).
//
// A CTA takes all 27 taps of a 16-channel slice of the input and 16 MB output channels, over a run
// of units (a unit: the 16 x 8 voxels of one brick of one plane z; z fastest), and keeps the
// accumulators in registers: warp (dz, dy) has the three taps dx, 9 warps.  What it stages is then
// its own channels once (the input planes z - 1, z, z + 1 in a ring of four, each fetched once a
// column by cp.async while the plane before is worked on), where a split by taps staged every
// channel of the halo in every group of taps and spent its time on that.  The masked gradient of
// the next unit comes through registers (two buffers).  One barrier a unit; a row of 16 voxels is
// one k-step: MB + 3 ldmatrix for 6 MB mma.
// 96 -> 32 at 64^3: 1618 -> 150 us; 16 -> 16 at 128^3: 290 -> 101 us (mma.sync's own limit is about
// a third of that).
constexpr int kWgThreads = 288;
constexpr int kPlaneVox = kHX * kHY;      // 180 voxels of a staged plane
constexpr int kXPitch = 48;               // bytes of a voxel's 16 channels, padded: conflict-free ldmatrix
constexpr int kXPlane = kPlaneVox * kXPitch;

template <int CIN, int COUT>
struct WGrad {
    static constexpr int MB = COUT >= 32 ? 2 : 1;        // 16-channel blocks of the output a CTA
    static constexpr int GROUPS = (CIN / 16) * (COUT / (16 * MB));
    static constexpr int GPITCH = 32 * MB + 16;          // bytes of a voxel's gradient slice, padded
    static constexpr int GTILE = 128 * GPITCH;
    static constexpr int SMEM = 4 * kXPlane + 2 * GTILE;
    static constexpr int CTAS = MB == 2 ? 2 : 3;         // resident per SM (registers)
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(kWgThreads, WGrad<CIN, COUT>::CTAS)
    conv3_wgrad_kernel(int X, int Y, int Z, ConvIn in, const __nv_bfloat16* __restrict__ g,
                       const __nv_bfloat16* __restrict__ y_out, int nsplit, float* __restrict__ part_w,
                       float* __restrict__ part_b) {
    using W = WGrad<CIN, COUT>;
    constexpr int MB = W::MB, GV = 2 * MB;  // 16-byte chunks of a voxel's gradient slice
    constexpr int kGPer = (128 * GV + kWgThreads - 1) / kWgThreads;  // gradient chunks a thread
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t xs = smem_u32(smem_raw), gs = xs + 4 * kXPlane;
    const int cis = blockIdx.x % (CIN / 16), cos = blockIdx.x / (CIN / 16), split = blockIdx.y;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int bx = (X + kTX - 1) / kTX, by = (Y + kTY - 1) / kTY;
    const long long units = (long long)bx * by * Z;
    const long long u_begin = units * split / nsplit, u_end = units * (split + 1) / nsplit;
    float acc[3][MB][2][4];
#pragma unroll
    for (int t = 0; t < 3; ++t)
#pragma unroll
        for (int m = 0; m < MB; ++m)
#pragma unroll
            for (int h = 0; h < 2; ++h) acc[t][m][h][0] = acc[t][m][h][1] = acc[t][m][h][2] = acc[t][m][h][3] = 0.f;
    float accb[MB][4];  // bias gradient (warp 0 of the first input slice): the row sums of gm^T
#pragma unroll
    for (int m = 0; m < MB; ++m) accb[m][0] = accb[m][1] = accb[m][2] = accb[m][3] = 0.f;
    const bool bias_warp = cis == 0 && warp == 0;

    int x0 = 0, y0 = 0;
    // chunk e of a plane: voxel e / 2, channels 8 (e % 2) of the slice; this thread's are tid and,
    // for the first 72 threads, tid + 288
    auto stage_plane = [&](int z) {
        const uint32_t slot = xs + (uint32_t)((z + 4) & 3) * kXPlane;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int e = tid + q * kWgThreads;
            if (e >= 2 * kPlaneVox) break;
            const int hv = e >> 1, hy = hv / kHX, hx = hv - hy * kHX;
            const int x = x0 + hx - 1, y = y0 + hy - 1, c = cis * 16 + (e & 1) * 8;
            const __nv_bfloat16* src = in.a;  // a valid address even when nothing is read
            bool valid = x >= 0 && x < X && y >= 0 && y < Y && z >= 0 && z < Z;
            if (valid) {
                if (c < in.ca) {
                    const long long v = in.up_a ? ((long long)(z >> 1) * in.ay + (y >> 1)) * in.ax + (x >> 1)
                                                : ((long long)z * Y + y) * X + x;
                    src = in.a + v * in.ca + c;
                } else if (in.b) {
                    src = in.b + (((long long)z * Y + y) * X + x) * in.cb + (c - in.ca);
                } else {
                    valid = false;
                }
            }
            cp_async16_zfill(slot + (uint32_t)(hv * kXPitch + (e & 1) * 16), src, valid);
        }
    };
    uint4 gr[kGPer], yr[kGPer];
    auto load_grad = [&](int z) {
#pragma unroll
        for (int q = 0; q < kGPer; ++q) {
            const int e = tid + q * kWgThreads, vv = e / GV, cv = e % GV;
            const int x = x0 + (vv & 15), y = y0 + (vv >> 4);
            gr[q] = yr[q] = make_uint4(0u, 0u, 0u, 0u);
            if (e < 128 * GV && x < X && y < Y) {
                const long long o = (((long long)z * Y + y) * X + x) * COUT + cos * 16 * MB + cv * 8;
                gr[q] = __ldg(reinterpret_cast<const uint4*>(g + o));
                yr[q] = __ldg(reinterpret_cast<const uint4*>(y_out + o));
            }
        }
    };
    auto store_grad = [&](int buf) {
#pragma unroll
        for (int q = 0; q < kGPer; ++q) {
            const int e = tid + q * kWgThreads;
            if (e < 128 * GV)
                *reinterpret_cast<uint4*>(smem_raw + 4 * kXPlane + buf * W::GTILE + (e / GV) * W::GPITCH + (e % GV) * 16) =
                    apply_relu_mask(gr[q], yr[q]);
        }
    };

    const int r = lane & 7, m4 = lane >> 3;
    const int dz = warp / 3 - 1, dy = warp % 3 - 1;
    // this lane's ldmatrix rows: A = gm^T (v 0-7|co 0-7), (v 0-7|co 8-15), (v 8-15|co 0-7), (v 8-15|co 8-15);
    // B = x shifted (v 0-7|ci 0-7), (v 8-15|ci 0-7), (v 0-7|ci 8-15), (v 8-15|ci 8-15)
    const uint32_t a_lane = (uint32_t)((r + (m4 >> 1) * 8) * W::GPITCH + (m4 & 1) * 16);
    const uint32_t b_lane = (uint32_t)(((1 + dy) * kHX + r + (m4 & 1) * 8) * kXPitch + (m4 >> 1) * 16);
    int buf = 0;
#pragma unroll 1
    for (long long u = u_begin; u < u_end; ++u) {
        const int z = (int)(u % Z);
        if (u == u_begin || z == 0) {  // a column begins: its first three planes and its first gradient
            __syncthreads();           // the unit before is done with the buffers
            const long long col = u / Z;
            x0 = (int)(col % bx) * kTX;
            y0 = (int)(col / bx) * kTY;
            stage_plane(z - 1);
            stage_plane(z);
            stage_plane(z + 1);
            load_grad(z);
            store_grad(buf);
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        const bool more = u + 1 < u_end && z + 1 < Z;  // the next unit continues this column
        if (more) {
            stage_plane(z + 2);
            load_grad(z + 1);
        }
        const uint32_t xp = xs + (uint32_t)((z + dz + 4) & 3) * kXPlane + b_lane;
        const uint32_t gp = gs + (uint32_t)(buf * W::GTILE) + a_lane;
#pragma unroll
        for (int row = 0; row < kTY; ++row) {
            uint32_t a[MB][4];
#pragma unroll
            for (int m = 0; m < MB; ++m) ldsm_x4_t(gp + (uint32_t)(row * 16 * W::GPITCH + m * 32), a[m]);
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                uint32_t b[4];
                ldsm_x4_t(xp + (uint32_t)((row * kHX + t) * kXPitch), b);
#pragma unroll
                for (int m = 0; m < MB; ++m) {
                    mma_bf16(acc[t][m][0], a[m], b[0], b[1]);
                    mma_bf16(acc[t][m][1], a[m], b[2], b[3]);
                }
            }
            if (bias_warp) {
#pragma unroll
                for (int m = 0; m < MB; ++m) mma_bf16(accb[m], a[m], 0x3f803f80u, 0x3f803f80u);  // times ones
            }
        }
        buf ^= 1;
        if (more) store_grad(buf);
    }
    // partial [split][tap][co][ci]
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        float* dst = part_w + ((size_t)split * 27 + warp * 3 + t) * COUT * CIN;
#pragma unroll
        for (int m = 0; m < MB; ++m)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int ci = cis * 16 + h * 8 + (lane & 3) * 2, co = (cos * MB + m) * 16 + (lane >> 2);
                // (one float a store: the caller's workspace need not be aligned for two)
                dst[(size_t)co * CIN + ci] = acc[t][m][h][0];
                dst[(size_t)co * CIN + ci + 1] = acc[t][m][h][1];
                dst[(size_t)(co + 8) * CIN + ci] = acc[t][m][h][2];
                dst[(size_t)(co + 8) * CIN + ci + 1] = acc[t][m][h][3];
            }
    }
    if (bias_warp && (lane & 3) == 0) {
#pragma unroll
        for (int m = 0; m < MB; ++m) {
            const int co = (cos * MB + m) * 16 + (lane >> 2);
            part_b[(size_t)split * COUT + co] = accb[m][0];
            part_b[(size_t)split * COUT + co + 8] = accb[m][2];
        }
    }
}

// dW[co][tap][ci] += sum over splits, db[co] += likewise, in a fixed order: a block takes 32 values,
// warp w sums every eighth split from w on, and the eight sums are added in order (a thread a value
// and all its splits in sequence left 28 blocks waiting for one load after another: 26 -> 6 us
// for 16 -> 16 at 128^3)
__global__ void __launch_bounds__(256) wgrad_reduce_kernel(int cin, int cout, int nsplit,
                                                           const float* __restrict__ part_w,
                                                           const float* __restrict__ part_b, float* __restrict__ dw,
                                                           float* __restrict__ db) {
    __shared__ float sums[8][32];
    const int per = 27 * cout * cin;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int e = blockIdx.x * 32 + lane;
    const float* p = e < per ? part_w + e : part_b + (e - per);
    const size_t stride = e < per ? (size_t)per : (size_t)cout;
    float s = 0.f;
    if (e < per + (db ? cout : 0)) {
#pragma unroll 8
        for (int q = warp; q < nsplit; q += 8) s += p[(size_t)q * stride];
    }
    sums[warp][lane] = s;
    __syncthreads();
    if (warp != 0) return;
#pragma unroll
    for (int q = 1; q < 8; ++q) s += sums[q][lane];
    if (e < per) {
        // e indexes the partial layout [tap][co][ci]; dW is [co][tap][ci]
        const int ci = e % cin, t2 = e / cin, co = t2 % cout, tap = t2 / cout;
        dw[((size_t)co * 27 + tap) * cin + ci] += s;
    } else if (db && e < per + cout) {
        db[e - per] += s;
    }
}

// ---------------------------------------------------------------------------------------
// weights: FP32 master [co][27][ci] -> bf16 B fragments for the forward (K = ci) and for the
// backward data pass (the transposed, tap-mirrored kernel, K = co)
__device__ __forceinline__ size_t frag_index(int tap, int n, int k, int kdim, int ndim) {
    const int ks = k >> 4, kk = k & 15, nb = n >> 3, nn = n & 7;
    const int ln = nn * 4 + ((kk & 7) >> 1);
    const int comp = (nb & 1) * 2 + (kk >> 3);
    const size_t u4 = (((size_t)tap * (kdim / 16) + ks) * (ndim / 16) + (nb >> 1)) * 32 + ln;
    return (u4 * 4 + comp) * 2 + (kk & 1);
}

__global__ void pack_weights_kernel(int cin, int cout, const float* __restrict__ w, __nv_bfloat16* __restrict__ wf,
                                    __nv_bfloat16* __restrict__ wb) {
    const long long n = 27LL * cin * cout;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const int ci = (int)(e % cin);
        const long long t2 = e / cin;
        const int tap = (int)(t2 % 27), co = (int)(t2 / 27);
        const __nv_bfloat16 v = __float2bfloat16_rn(w[e]);
        wf[frag_index(tap, co, ci, cin, cout)] = v;
        if (wb) wb[frag_index(26 - tap, ci, co, cout, cin)] = v;
    }
}

// ---------------------------------------------------------------------------------------
// 2x2x2 average pooling, its backward (accumulated into the fine gradient) and the backward
// of nearest upsampling (sum of the 8 children); 8 channels per thread
__global__ void pool_fwd_kernel(int X, int Y, int Z, int C, const __nv_bfloat16* __restrict__ in,
                                __nv_bfloat16* __restrict__ out) {
    const int Xc = X / 2, Yc = Y / 2, Zc = Z / 2, CV = C / 8;
    const long long n = (long long)Xc * Yc * Zc * CV;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const int cv = (int)(e % CV);
        const long long V = e / CV;
        const int xc = (int)(V % Xc), yc = (int)((V / Xc) % Yc), zc = (int)(V / ((long long)Xc * Yc));
        float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int q = 0; q < 8; ++q) {
            const long long v = ((long long)(2 * zc + (q >> 2)) * Y + 2 * yc + ((q >> 1) & 1)) * X + 2 * xc + (q & 1);
            const uint4 u = __ldg(reinterpret_cast<const uint4*>(in + v * C + cv * 8));
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = __bfloat1622float2(h[j]);
                s[2 * j] += f.x;
                s[2 * j + 1] += f.y;
            }
        }
        uint4 o;
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(s[2 * j] * 0.125f, s[2 * j + 1] * 0.125f);
        *reinterpret_cast<uint4*>(out + V * C + cv * 8) = o;
    }
}

// fine[v] (+)= scale * coarse[v / 2]: pooling backward (scale 1/8, accumulate)
__global__ void spread_kernel(int X, int Y, int Z, int C, const __nv_bfloat16* __restrict__ coarse,
                              __nv_bfloat16* __restrict__ fine, float scale, int accumulate) {
    const int CV = C / 8, Xc = X / 2, Yc = Y / 2;
    const long long n = (long long)X * Y * Z * CV;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const int cv = (int)(e % CV);
        const long long v = e / CV;
        const int x = (int)(v % X), y = (int)((v / X) % Y), z = (int)(v / ((long long)X * Y));
        const long long V = ((long long)(z >> 1) * Yc + (y >> 1)) * Xc + (x >> 1);
        const uint4 cu = __ldg(reinterpret_cast<const uint4*>(coarse + V * C + cv * 8));
        const __nv_bfloat162* ch = reinterpret_cast<const __nv_bfloat162*>(&cu);
        uint4* fp = reinterpret_cast<uint4*>(fine + v * C + cv * 8);
        uint4 fu = accumulate ? *fp : make_uint4(0u, 0u, 0u, 0u);
        __nv_bfloat162* fh = reinterpret_cast<__nv_bfloat162*>(&fu);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 c2 = __bfloat1622float2(ch[j]);
            const float2 f2 = accumulate ? __bfloat1622float2(fh[j]) : make_float2(0.f, 0.f);
            fh[j] = __floats2bfloat162_rn(f2.x + scale * c2.x, f2.y + scale * c2.y);
        }
        *fp = fu;
    }
}

// coarse[V] = sum of the 8 fine children: backward of nearest upsampling
__global__ void gather8_kernel(int X, int Y, int Z, int C, const __nv_bfloat16* __restrict__ fine,
                               __nv_bfloat16* __restrict__ coarse) {
    const int Xc = X / 2, Yc = Y / 2, Zc = Z / 2, CV = C / 8;
    const long long n = (long long)Xc * Yc * Zc * CV;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const int cv = (int)(e % CV);
        const long long V = e / CV;
        const int xc = (int)(V % Xc), yc = (int)((V / Xc) % Yc), zc = (int)(V / ((long long)Xc * Yc));
        float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int q = 0; q < 8; ++q) {
            const long long v = ((long long)(2 * zc + (q >> 2)) * Y + 2 * yc + ((q >> 1) & 1)) * X + 2 * xc + (q & 1);
            const uint4 u = __ldg(reinterpret_cast<const uint4*>(fine + v * C + cv * 8));
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = __bfloat1622float2(h[j]);
                s[2 * j] += f.x;
                s[2 * j + 1] += f.y;
            }
        }
        uint4 o;
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(s[2 * j], s[2 * j + 1]);
        *reinterpret_cast<uint4*>(coarse + V * C + cv * 8) = o;
    }
}

// ---------------------------------------------------------------------------------------
// head: pred = w . d + b (16 channels -> 1, FP32)
constexpr int kHeadC = 16;

__global__ void head_fwd_kernel(long long n, const __nv_bfloat16* __restrict__ d, const float* __restrict__ w,
                                const float* __restrict__ b, float* __restrict__ pred) {
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        const uint4* p = reinterpret_cast<const uint4*>(d + v * kHeadC);
        float s = b[0];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint4 u = __ldg(p + h);
            const __nv_bfloat162* q = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = __bfloat1622float2(q[j]);
                s += w[h * 8 + 2 * j] * f.x + w[h * 8 + 2 * j + 1] * f.y;
            }
        }
        pred[v] = s;
    }
}

// Masked mean-square loss and the head's backward: e = pred - target on cells with mask != 0,
// loss += e^2 * inv_n, g = 2 e inv_n, grad_d = g w (bf16), dw += g d, db += g.  Totals by a
// deterministic grid reduction, added to loss (FP64) and to the head's FP32 gradients.
__global__ void head_loss_bwd_kernel(long long n, const __nv_bfloat16* __restrict__ d, const float* __restrict__ pred,
                                     const float* __restrict__ target, const uint8_t* __restrict__ mask,
                                     const float* __restrict__ w, double inv_n, __nv_bfloat16* __restrict__ grad_d,
                                     double* __restrict__ loss, float* __restrict__ dw, float* __restrict__ db,
                                     double* partials, unsigned* counter) {
    double acc[18];
#pragma unroll
    for (int q = 0; q < 18; ++q) acc[q] = 0.0;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        float gv = 0.f;
        if (mask[v]) {
            const float e = pred[v] - target[v];
            acc[0] += (double)e * e * inv_n;
            gv = (float)(2.0 * inv_n) * e;
        }
        const uint4* p = reinterpret_cast<const uint4*>(d + v * kHeadC);
        uint4* o = reinterpret_cast<uint4*>(grad_d + v * kHeadC);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint4 u = __ldg(p + h);
            const __nv_bfloat162* q = reinterpret_cast<const __nv_bfloat162*>(&u);
            uint4 go;
            __nv_bfloat162* gq = reinterpret_cast<__nv_bfloat162*>(&go);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = __bfloat1622float2(q[j]);
                const int c = h * 8 + 2 * j;
                acc[1 + c] += (double)gv * f.x;
                acc[2 + c] += (double)gv * f.y;
                gq[j] = __floats2bfloat162_rn(gv * w[c], gv * w[c + 1]);
            }
            o[h] = go;
        }
        acc[17] += gv;
    }
    double tot[18];
    if (grid_sum<18>(acc, partials, counter, tot)) {
        loss[0] += tot[0];
#pragma unroll
        for (int q = 0; q < kHeadC; ++q) dw[q] += (float)tot[1 + q];
        db[0] += (float)tot[17];
    }
}

// Energy-norm loss and the head's backward.  With e = pred - target on fluid cells and A^ the
// scaled operator in Laplacian form (per cell: the diagonal excess delta and the face weights w
// with +x, +y, +z, all >= 0), the loss is e . A^ e * inv_n = (sum_faces w (e_c - e_n)^2 +
// sum delta e^2) * inv_n -- the error in the norm that conjugate gradients minimises, positive
// whatever the rounding of the weights -- and its gradient 2 (A^ e) inv_n with
// (A^ e)_c = delta e_c + sum_n w (e_c - e_n).  The rest as head_loss_bwd_kernel.
__device__ __forceinline__ float4 load_coup(const __nv_bfloat16* coup, long long v) {
    const uint2 q = __ldg(reinterpret_cast<const uint2*>(coup + v * 4));
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
    const float2 a = __bfloat1622float2(h[0]), b = __bfloat1622float2(h[1]);
    return make_float4(a.x, a.y, b.x, b.y);
}

__global__ void head_energy_bwd_kernel(int X, int Y, int Z, const __nv_bfloat16* __restrict__ d,
                                       const float* __restrict__ pred, const float* __restrict__ target,
                                       const __nv_bfloat16* __restrict__ coup, const uint8_t* __restrict__ fluid,
                                       const float* __restrict__ w,
                                       double inv_n, __nv_bfloat16* __restrict__ grad_d, double* __restrict__ loss,
                                       float* __restrict__ dw, float* __restrict__ db, double* partials,
                                       unsigned* counter) {
    const long long n = (long long)X * Y * Z;
    const long long sy = X, sz = (long long)X * Y;
    double acc[18];
#pragma unroll
    for (int q = 0; q < 18; ++q) acc[q] = 0.0;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(v % X), y = (int)((v / X) % Y), z = (int)(v / sz);
        const float4 cv = load_coup(coup, v);
        float gv = 0.f;
        if (fluid[v]) {
            const float e = pred[v] - target[v];
            float r = cv.x * e;                     // delta e
            double en = (double)cv.x * e * e;       // this cell's share of the energy: delta e^2
            auto face = [&](float w, long long q) { // a face to a fluid neighbour (w > 0 only then)
                if (w != 0.f) {
                    const float de = e - (pred[q] - target[q]);
                    r += w * de;
                    en += 0.5 * (double)w * de * de;  // each face is seen from both cells
                }
            };
            if (x + 1 < X) face(cv.y, v + 1);
            if (y + 1 < Y) face(cv.z, v + sy);
            if (z + 1 < Z) face(cv.w, v + sz);
            if (x > 0) face(load_coup(coup, v - 1).y, v - 1);
            if (y > 0) face(load_coup(coup, v - sy).z, v - sy);
            if (z > 0) face(load_coup(coup, v - sz).w, v - sz);
            acc[0] += en * inv_n;
            gv = (float)(2.0 * inv_n) * r;
        }
        const uint4* p = reinterpret_cast<const uint4*>(d + v * kHeadC);
        uint4* o = reinterpret_cast<uint4*>(grad_d + v * kHeadC);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint4 u = __ldg(p + h);
            const __nv_bfloat162* q = reinterpret_cast<const __nv_bfloat162*>(&u);
            uint4 go;
            __nv_bfloat162* gq = reinterpret_cast<__nv_bfloat162*>(&go);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = __bfloat1622float2(q[j]);
                const int c = h * 8 + 2 * j;
                acc[1 + c] += (double)gv * f.x;
                acc[2 + c] += (double)gv * f.y;
                gq[j] = __floats2bfloat162_rn(gv * w[c], gv * w[c + 1]);
            }
            o[h] = go;
        }
        acc[17] += gv;
    }
    double tot[18];
    if (grid_sum<18>(acc, partials, counter, tot)) {
        loss[0] += tot[0];
#pragma unroll
        for (int q = 0; q < kHeadC; ++q) dw[q] += (float)tot[1 + q];
        db[0] += (float)tot[17];
    }
}

// Adam on FP32 parameters; the gradient is zeroed for the next accumulation.
__global__ void adam_kernel(long long n, float* __restrict__ w, float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const float ge = g[e];
        const float me = b1 * m[e] + (1.f - b1) * ge;
        const float ve = b2 * v[e] + (1.f - b2) * ge * ge;
        m[e] = me;
        v[e] = ve;
        w[e] -= lr * (me * c1) / (sqrtf(ve * c2) + eps);
        g[e] = 0.f;
    }
}

}  // namespace nn
}  // namespace el

// =========================================================================================
// host side: launchers and the C ABI (include/eulerian_liquid_gb300.h, "learned warm start")
#include <algorithm>

using namespace el;
using namespace el::nn;

namespace {

int num_sms_current() {
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

int grid_elems(long long n) { return (int)std::max<long long>(1, std::min<long long>((n + 255) / 256, 152LL * 16)); }

ConvIn conv_in(const el_nn_conv_args* a) {
    ConvIn in;
    in.a = static_cast<const __nv_bfloat16*>(a->in_a);
    in.b = static_cast<const __nv_bfloat16*>(a->in_b);
    in.mask = static_cast<const __nv_bfloat16*>(a->mask);
    in.ca = a->ca;
    in.cb = a->cb;
    in.up_a = a->upsample_a;
    in.ax = a->upsample_a ? a->nx / 2 : a->nx;
    in.ay = a->upsample_a ? a->ny / 2 : a->ny;
    in.az = a->upsample_a ? a->nz / 2 : a->nz;
    return in;
}

template <int CIN, int COUT>
int launch_conv(const el_nn_conv_args* a, cudaStream_t s) {
    const size_t smem = (size_t)kHV * (CIN + 8) * sizeof(__nv_bfloat16);
    if (cudaFuncSetAttribute(conv3_kernel<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
        return EL_ERR_CUDA;
    const dim3 grid((a->nx + kTX - 1) / kTX, (a->ny + kTY - 1) / kTY, a->nz);
    conv3_kernel<CIN, COUT><<<grid, kThreads, smem, s>>>(
        a->nx, a->ny, a->nz, conv_in(a), static_cast<const uint4*>(a->weights), a->bias, a->relu,
        static_cast<__nv_bfloat16*>(a->out_a), a->out_a_channels, static_cast<__nv_bfloat16*>(a->out_b));
    return cudaGetLastError() == cudaSuccess ? EL_OK : EL_ERR_CUDA;
}

template <int CIN, int COUT, int SC, int CTAS>
int launch_conv_tc(const el_nn_conv_args* a, cudaStream_t s) {
    using SS = tc::RunShape<CIN, COUT, SC, CTAS>;
    if (cudaFuncSetAttribute(tc::conv3_tc_kernel<CIN, COUT, SC, CTAS>, cudaFuncAttributePreferredSharedMemoryCarveout,
                             (int)cudaSharedmemCarveoutMaxShared) != cudaSuccess)
        return EL_ERR_CUDA;
    if (cudaFuncSetAttribute(tc::conv3_tc_kernel<CIN, COUT, SC, CTAS>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, SS::S::SMEM) != cudaSuccess)
        return EL_ERR_CUDA;
    const long long units = (long long)((a->nx + tc::TX - 1) / tc::TX) * ((a->ny + tc::TY - 1) / tc::TY) * a->nz;
    const int grid = (int)std::min<long long>(units, (long long)num_sms_current() * CTAS);
    tc::conv3_tc_kernel<CIN, COUT, SC, CTAS><<<grid, tc::kThreads, SS::S::SMEM, s>>>(
        a->nx, a->ny, a->nz, conv_in(a), static_cast<const uint4*>(a->weights_tc), a->bias, a->relu,
        static_cast<__nv_bfloat16*>(a->out_a), a->out_a_channels, static_cast<__nv_bfloat16*>(a->out_b));
    return cudaGetLastError() == cudaSuccess ? EL_OK : EL_ERR_CUDA;
}

// one wave of resident CTAs over the channel slices, at most a split a unit
template <int CIN, int COUT>
int wgrad_splits(int nx, int ny, int nz) {
    const long long units = (long long)((nx + kTX - 1) / kTX) * ((ny + kTY - 1) / kTY) * nz;
    const int want = WGrad<CIN, COUT>::CTAS * num_sms_current() / WGrad<CIN, COUT>::GROUPS;
    return (int)std::max<long long>(1, std::min<long long>(want, units));
}

template <int CIN, int COUT>
size_t wgrad_ws(int nx, int ny, int nz) {
    const int ns = wgrad_splits<CIN, COUT>(nx, ny, nz);
    return ((size_t)ns * 27 * CIN * COUT + (size_t)ns * COUT) * sizeof(float);
}

template <int CIN, int COUT>
int launch_wgrad(const el_nn_conv_args* a, const void* grad_out, float* dw, float* db, void* ws, size_t ws_bytes,
                 cudaStream_t s) {
    using W = WGrad<CIN, COUT>;
    const int ns = wgrad_splits<CIN, COUT>(a->nx, a->ny, a->nz);
    if (ws_bytes < wgrad_ws<CIN, COUT>(a->nx, a->ny, a->nz)) return EL_ERR_INVALID_ARGUMENT;
    float* part_w = static_cast<float*>(ws);
    float* part_b = part_w + (size_t)ns * 27 * CIN * COUT;
    if (cudaFuncSetAttribute(conv3_wgrad_kernel<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, W::SMEM) !=
        cudaSuccess)
        return EL_ERR_CUDA;
    conv3_wgrad_kernel<CIN, COUT><<<dim3(W::GROUPS, ns), kWgThreads, W::SMEM, s>>>(
        a->nx, a->ny, a->nz, conv_in(a), static_cast<const __nv_bfloat16*>(grad_out),
        static_cast<const __nv_bfloat16*>(a->out_a), ns, part_w, part_b);
    const int n = 27 * CIN * COUT + COUT;
    wgrad_reduce_kernel<<<(n + 31) / 32, 256, 0, s>>>(CIN, COUT, ns, part_w, part_b, dw, db);
    return cudaGetLastError() == cudaSuccess ? EL_OK : EL_ERR_CUDA;
}

// (cin, cout) pairs of the network, forward and backward-data
#define EL_NN_CONV_PAIRS(X)                                                                                      \
    X(16, 16) X(16, 32) X(32, 32) X(32, 64) X(64, 64) X(128, 64) X(96, 32) X(48, 16) X(32, 16) X(64, 32) X(64, 128) \
        X(32, 96) X(16, 48)
// the same on the tcgen05 kernel: input channels a slice, resident CTAs an SM (the fastest of the
// combinations that fit, over the layers' grids; e.g. 32 -> 32 at 64^3 in slices of 16, three CTAs: 41 us
// against 31; 96 -> 32 in slices of 16, three CTAs: 100 against 75; 64 -> 32 at 32^3: 22.7 against 18.6)
#define EL_NN_TC_PAIRS(X)                                                                                    \
    X(16, 16, 16, 4) X(16, 32, 16, 4) X(32, 32, 32, 2) X(32, 64, 32, 1) X(64, 64, 32, 1) X(128, 64, 32, 1)   \
        X(96, 32, 32, 2) X(48, 16, 16, 4) X(32, 16, 32, 2) X(64, 32, 32, 2) X(64, 128, 16, 1) X(32, 96, 32, 1) \
        X(16, 48, 16, 3)
// forward pairs (backward weight)
#define EL_NN_FWD_PAIRS(X) X(16, 16) X(16, 32) X(32, 32) X(32, 64) X(64, 64) X(128, 64) X(96, 32) X(48, 16)

bool valid_conv(const el_nn_conv_args* a) {
    if (!a || a->nx < 1 || a->ny < 1 || a->nz < 1 || a->ca < 0 || a->cb < 0 || a->ca % 8 || a->cb % 8 ||
        a->ca + a->cb != a->cin || !a->in_a)
        return false;
    if (a->upsample_a && (a->nx % 2 || a->ny % 2 || a->nz % 2)) return false;
    return true;
}

}  // namespace

#define EL_API extern "C" __attribute__((visibility("default")))

EL_API int el_nn_tc_supported(int cin, int cout) {
#define EL_NN_CASE(CI, CO, SC, CTAS) \
    if (cin == CI && cout == CO) return 1;
    EL_NN_TC_PAIRS(EL_NN_CASE)
#undef EL_NN_CASE
    return 0;
}

// Every pair: no layer of the network measured slower on the tcgen05 kernel than on the mma.sync one
// (us, mma.sync / tcgen05: 16 -> 16 at 128^3 230 / 88, 48 -> 16 664 / 222, 16 -> 48 363 / 188; at 64^3
// 32 -> 32 65 / 31, 96 -> 32 212 / 75; at 32^3 64 -> 64 34 / 21, 128 -> 64 106 / 33, 16 -> 32 10.5 / 8.4;
// at 8^3 64 -> 64 29 / 13).
EL_API int el_nn_tc_preferred(int cin, int cout) { return el_nn_tc_supported(cin, cout); }

EL_API int el_nn_take_error(void) {
    int e = 0;
    const int zero = 0;
    if (cudaMemcpyFromSymbol(&e, tc::g_error, sizeof(int)) != cudaSuccess) return -1;
    if (e && cudaMemcpyToSymbol(tc::g_error, &zero, sizeof(int)) != cudaSuccess) return -1;
    return e;
}

EL_API int el_nn_conv3_forward(const el_nn_conv_args* a, void* stream) {
    if (a && a->weights_tc && el_nn_tc_supported(a->cin, a->cout) && valid_conv(a) && a->out_a &&
        a->out_a_channels > 0 && a->out_a_channels <= a->cout && a->out_a_channels % 8 == 0 &&
        (a->out_a_channels == a->cout || a->out_b)) {
        cudaStream_t s = static_cast<cudaStream_t>(stream);
#define EL_NN_CASE(CI, CO, SC, CTAS) \
        if (a->cin == CI && a->cout == CO) return launch_conv_tc<CI, CO, SC, CTAS>(a, s);
        EL_NN_TC_PAIRS(EL_NN_CASE)
#undef EL_NN_CASE
    }
    if (!valid_conv(a) || !a->weights || !a->out_a || a->out_a_channels <= 0 || a->out_a_channels > a->cout ||
        a->out_a_channels % 8 || (a->out_a_channels < a->cout && !a->out_b))
        return EL_ERR_INVALID_ARGUMENT;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
#define EL_NN_CASE(CI, CO) \
    if (a->cin == CI && a->cout == CO) return launch_conv<CI, CO>(a, s);
    EL_NN_CONV_PAIRS(EL_NN_CASE)
#undef EL_NN_CASE
    return EL_ERR_INVALID_ARGUMENT;
}

EL_API size_t el_nn_conv3_backward_weight_workspace(int nx, int ny, int nz, int cin, int cout) {
#define EL_NN_CASE(CI, CO) \
    if (cin == CI && cout == CO) return wgrad_ws<CI, CO>(nx, ny, nz);
    EL_NN_FWD_PAIRS(EL_NN_CASE)
#undef EL_NN_CASE
    return 0;
}

EL_API int el_nn_conv3_backward_weight(const el_nn_conv_args* a, const void* grad_out, float* dw, float* db,
                                       void* workspace, size_t workspace_bytes, void* stream) {
    if (!valid_conv(a) || !a->out_a || !grad_out || !dw || !workspace) return EL_ERR_INVALID_ARGUMENT;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
#define EL_NN_CASE(CI, CO) \
    if (a->cin == CI && a->cout == CO) return launch_wgrad<CI, CO>(a, grad_out, dw, db, workspace, workspace_bytes, s);
    EL_NN_FWD_PAIRS(EL_NN_CASE)
#undef EL_NN_CASE
    return EL_ERR_INVALID_ARGUMENT;
}

EL_API size_t el_nn_packed_weight_bytes(int cin, int cout) { return (size_t)27 * cin * cout * sizeof(__nv_bfloat16); }

EL_API int el_nn_pack_weights(int cin, int cout, const float* w, void* packed_fwd, void* packed_bwd, void* stream) {
    if (cin % 16 || cout % 16 || cin <= 0 || cout <= 0 || !w || !packed_fwd) return EL_ERR_INVALID_ARGUMENT;
    const long long n = 27LL * cin * cout;
    pack_weights_kernel<<<grid_elems(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        cin, cout, w, static_cast<__nv_bfloat16*>(packed_fwd), static_cast<__nv_bfloat16*>(packed_bwd));
    return cudaGetLastError() == cudaSuccess ? EL_OK : EL_ERR_CUDA;
}

EL_API int el_nn_pack_weights_tc(int cin, int cout, const float* w, void* packed_fwd, void* packed_bwd,
                                  void* stream) {
    if (cin % 16 || cout % 16 || cin <= 0 || cout <= 0 || !w || !packed_fwd) return EL_ERR_INVALID_ARGUMENT;
    const long long n = 27LL * cin * cout;
    tc::pack_weights_tc_kernel<<<grid_elems(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        cin, cout, w, static_cast<__nv_bfloat16*>(packed_fwd), static_cast<__nv_bfloat16*>(packed_bwd));
    return cudaGetLastError() == cudaSuccess ? EL_OK : EL_ERR_CUDA;
}

EL_API int el_nn_pool(int nx, int ny, int nz, int c, const void* in, void* out, void* stream) {
    if (nx % 2 || ny % 2 || nz % 2 || c % 8 || !in || !out) return EL_ERR_INVALID_ARGUMENT;
    const long long n = (long long)(nx / 2) * (ny / 2) * (nz / 2) * (c / 8);
    pool_fwd_kernel<<<grid_elems(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        nx, ny, nz, c, static_cast<const __nv_bfloat16*>(in), static_cast<__nv_bfloat16*>(out));
    return cudaGetLastError() == cudaSuccess ? EL_OK : EL_ERR_CUDA;
}

EL_API int el_nn_spread(int nx, int ny, int nz, int c, const void* coarse, void* fine, float scale, int accumulate,
                        void* stream) {
    if (nx % 2 || ny % 2 || nz % 2 || c % 8 || !coarse || !fine) return EL_ERR_INVALID_ARGUMENT;
    const long long n = (long long)nx * ny * nz * (c / 8);
    spread_kernel<<<grid_elems(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        nx, ny, nz, c, static_cast<const __nv_bfloat16*>(coarse), static_cast<__nv_bfloat16*>(fine), scale, accumulate);
    return cudaGetLastError() == cudaSuccess ? EL_OK : EL_ERR_CUDA;
}

EL_API int el_nn_gather8(int nx, int ny, int nz, int c, const void* fine, void* coarse, void* stream) {
    if (nx % 2 || ny % 2 || nz % 2 || c % 8 || !coarse || !fine) return EL_ERR_INVALID_ARGUMENT;
    const long long n = (long long)(nx / 2) * (ny / 2) * (nz / 2) * (c / 8);
    gather8_kernel<<<grid_elems(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        nx, ny, nz, c, static_cast<const __nv_bfloat16*>(fine), static_cast<__nv_bfloat16*>(coarse));
    return cudaGetLastError() == cudaSuccess ? EL_OK : EL_ERR_CUDA;
}

EL_API int el_nn_head_forward(int64_t n, const void* d, const float* w, const float* b, float* pred, void* stream) {
    if (n < 0 || !d || !w || !b || !pred) return EL_ERR_INVALID_ARGUMENT;
    head_fwd_kernel<<<grid_elems(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        n, static_cast<const __nv_bfloat16*>(d), w, b, pred);
    return cudaGetLastError() == cudaSuccess ? EL_OK : EL_ERR_CUDA;
}

EL_API size_t el_nn_head_workspace(int64_t n) { return (size_t)grid_elems(n) * 18 * sizeof(double) + 64; }

EL_API int el_nn_head_loss_backward(int64_t n, const void* d, const float* pred, const float* target,
                                    const uint8_t* mask, const float* w, double inv_n, void* grad_d, double* loss,
                                    float* dw, float* db, void* workspace, size_t workspace_bytes, void* stream) {
    if (n < 0 || !d || !pred || !target || !mask || !w || !grad_d || !loss || !dw || !db || !workspace ||
        workspace_bytes < el_nn_head_workspace(n))
        return EL_ERR_INVALID_ARGUMENT;
    const int blocks = grid_elems(n);
    double* partials = static_cast<double*>(workspace);
    unsigned* counter = reinterpret_cast<unsigned*>(static_cast<char*>(workspace) + (size_t)blocks * 18 * sizeof(double));
    head_loss_bwd_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        n, static_cast<const __nv_bfloat16*>(d), pred, target, mask, w, inv_n, static_cast<__nv_bfloat16*>(grad_d),
        loss, dw, db, partials, counter);
    return cudaGetLastError() == cudaSuccess ? EL_OK : EL_ERR_CUDA;
}

EL_API int el_nn_head_energy_loss_backward(int nx, int ny, int nz, const void* d, const float* pred,
                                           const float* target, const void* couplings, const uint8_t* fluid,
                                           const float* w, double inv_n, void* grad_d, double* loss, float* dw,
                                           float* db, void* workspace, size_t workspace_bytes, void* stream) {
    const int64_t n = (int64_t)nx * ny * nz;
    if (nx < 1 || ny < 1 || nz < 1 || !d || !pred || !target || !couplings || !fluid || !w || !grad_d || !loss ||
        !dw || !db ||
        !workspace || workspace_bytes < el_nn_head_workspace(n))
        return EL_ERR_INVALID_ARGUMENT;
    const int blocks = grid_elems(n);
    double* partials = static_cast<double*>(workspace);
    unsigned* counter = reinterpret_cast<unsigned*>(static_cast<char*>(workspace) + (size_t)blocks * 18 * sizeof(double));
    head_energy_bwd_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        nx, ny, nz, static_cast<const __nv_bfloat16*>(d), pred, target, static_cast<const __nv_bfloat16*>(couplings),
        fluid, w, inv_n, static_cast<__nv_bfloat16*>(grad_d), loss, dw, db, partials, counter);
    return cudaGetLastError() == cudaSuccess ? EL_OK : EL_ERR_CUDA;
}

EL_API int el_nn_adam(int64_t n, float* w, float* g, float* m, float* v, float lr, float beta1, float beta2,
                      float eps, int step, void* stream) {
    if (n < 0 || !w || !g || !m || !v || step < 1) return EL_ERR_INVALID_ARGUMENT;
    const float c1 = 1.f / (1.f - powf(beta1, (float)step));
    const float c2 = 1.f / (1.f - powf(beta2, (float)step));
    adam_kernel<<<grid_elems(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(n, w, g, m, v, lr, beta1, beta2, eps, c1,
                                                                              c2);
    return cudaGetLastError() == cudaSuccess ? EL_OK : EL_ERR_CUDA;
}
