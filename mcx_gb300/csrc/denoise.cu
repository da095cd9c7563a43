// Kernels of the fluence denoiser: a 4-level 3D U-Net (16/32/64/128 channels, 3x3x3 convolutions,
// ReLU, 2x2x2 average pooling, nearest upsampling with skip concatenation, a 1x1x1 head added to
// the input log-fluence) trained on pairs of low- and high-photon fluence maps from this engine.
//
// Layout: activations are channels-last bf16, [volumes][z][y][x][channels] with x fastest over
// voxels (MCX's own voxel order, so a fluence map is used in place); convolution weights are
// bf16 [Cout][taps][Cin] with tap = dz*9 + dy*3 + dx; master weights, gradients and Adam moments
// are fp32 in the same order.
//
// Convolutions are implicit GEMMs on the BF16 tensor cores, fp32 accumulate: the 3x3x3 ones forward and as data
// gradients on tcgen05 (conv3_roll.cuh), the weight gradient and what that kernel does not take on mma.sync m16n8k16:
//   forward   Y[v, co]  = sum_{t, ci} X[v + off(t), ci] * W[co, t, ci]      (M = voxels, N = Cout)
//   data grad dX[v, ci] = sum_{t, co} dY[v + off(t), co] * W[co, 26-t, ci] (the forward kernel run
//             on the flipped, transposed copy of W that the optimiser writes beside the weights)
//   weight gr dW[co, t, ci] = sum_v dY[v, co] * X[v + off(t), ci]         (M = Cout, N = taps*Cin,
//             K = voxels split across CTAs, fp32 atomics)
// Operand tiles are staged through a 4-deep cp.async pipeline into XOR-swizzled shared memory and
// fed to the tensor cores with ldmatrix (.trans for the weight gradient's voxel-major operands).
// Zero padding of the 3x3x3 stencil is the cp.async zero fill.  The ReLU backward is fused: a data
// gradient is multiplied by (layer input > 0) in its epilogue, so every gradient handed to a
// weight-gradient launch is already the pre-activation gradient.
#include <cuda_bf16.h>
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <stdint.h>

#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "mcxg_denoise.h"

namespace {

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// 16-byte asynchronous copy global -> shared; `valid` false copies nothing and fills zeros.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
    int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void ldsm_x4(uint32_t a, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t a, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Shared-memory tiles are rows of CPR 16-byte chunks; chunk c of row r is stored at
// c ^ swz(r) so that the 8 rows one ldmatrix phase reads fall in 8 different bank groups.
template <int CPR>
__device__ __forceinline__ int swz(int r) {
    if constexpr (CPR >= 8) return r & 7;
    else if constexpr (CPR == 4) return (r >> 1) & 3;
    else return (r >> 2) & 1;
}

struct Geo {
    int nvol, d, h, w;
    long long m;  // voxels over all volumes
};

// ---------------------------------------------------------------------------------------------
// Forward convolution (and data gradient): Y[v, n0:n0+BN] over a tile of BM voxels.  K runs over
// (tap, input channel) flattened, k = tap*cin + ci, in stages of BK: with few input channels one
// stage spans several taps (4 taps of 16 channels at BK = 64), so small layers still feed the
// tensor cores several k16 steps per barrier.  A chunk of 8 channels never straddles two taps
// (cin % 8 == 0); chunks past the last tap are zero-filled, as are the halo's out-of-volume rows.
template <int BM, int BN, int BK, int WARPS_M, int WARPS_N, int STAGES>
__global__ void __launch_bounds__(32 * WARPS_M * WARPS_N) conv_fwd_kernel(
    const bf16* __restrict__ x, const bf16* __restrict__ wt, const float* __restrict__ bias,
    const bf16* __restrict__ mask, bf16* __restrict__ y, Geo g, int cin, int cout, int taps, int relu) {
    constexpr int THREADS = 32 * WARPS_M * WARPS_N;
    constexpr int CPR = BK / 8;
    constexpr int WM = BM / WARPS_M, WN = BN / WARPS_N;
    constexpr int MI = WM / 16, NI = WN / 8;
    constexpr int A_ELEMS = BM * BK, B_ELEMS = BN * BK;
    constexpr int STAGE = A_ELEMS + B_ELEMS;
    constexpr int A_IT = BM * CPR / THREADS;
    static_assert(NI % 2 == 0 && MI >= 1 && A_IT >= 1 && (BM * CPR) % THREADS == 0 && THREADS % CPR == 0, "tile shape");

    extern __shared__ __align__(1024) unsigned char dyn_smem[];
    bf16* sm = reinterpret_cast<bf16*>(dyn_smem);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm0 = (warp / WARPS_N) * WM, wn0 = (warp % WARPS_N) * WN;
    const long long m0 = (long long)blockIdx.x * BM;
    const int n0 = blockIdx.y * BN;
    const int ktot = taps * cin;
    const int ktiles = (ktot + BK - 1) / BK;
    const int ac = tid % CPR;                      // the A chunk column this thread loads
    const int hw = g.h * g.w;

    // packed (z, y, x) of the tile's rows, one 32-bit decomposition per row shared through shared
    // memory (-1 past the last voxel); each thread keeps those of the A rows it loads
    __shared__ int s_zyx[BM];
    {
        const int vvol = g.d * hw;
        for (int r = tid; r < BM; r += THREADS) {
            long long v = m0 + r;
            int rr = (int)(v % vvol);
            int xx = rr % g.w, q = rr / g.w;
            s_zyx[r] = v < g.m ? (((q / g.h) << 20) | ((q % g.h) << 10) | xx) : -1;
        }
    }
    __syncthreads();
    int av[A_IT], azyx[A_IT];
#pragma unroll
    for (int i = 0; i < A_IT; ++i) {
        int row = tid / CPR + i * (THREADS / CPR);
        azyx[i] = s_zyx[row];
        av[i] = azyx[i] >= 0 ? (int)(m0 + row) : -1;
    }

    auto load_stage = [&](int stage, int kt) {
        bf16* sa = sm + stage * STAGE;
        bf16* sb = sa + A_ELEMS;
        const int k = kt * BK + ac * 8;
        const int t = k / cin, ch = k - t * cin;
        int dz = 0, dy = 0, dx = 0;
        if (taps == 27) {
            dz = t / 9 - 1;
            dy = (t / 3) % 3 - 1;
            dx = t % 3 - 1;
        }
        const bool kin = t < taps;
        const int delta = dz * hw + dy * g.w + dx;
#pragma unroll
        for (int i = 0; i < A_IT; ++i) {
            int row = tid / CPR + i * (THREADS / CPR);
            int zz = (azyx[i] >> 20) + dz, yy = ((azyx[i] >> 10) & 1023) + dy, xx = (azyx[i] & 1023) + dx;
            bool ok = kin && av[i] >= 0 && zz >= 0 && zz < g.d && yy >= 0 && yy < g.h && xx >= 0 && xx < g.w;
            const bf16* p = ok ? x + (long long)(av[i] + delta) * cin + ch : x;
            cp_async16(smem_addr(sa + row * BK + ((ac ^ swz<CPR>(row)) << 3)), p, ok);
        }
#pragma unroll
        for (int i = 0; i < (BN * CPR + THREADS - 1) / THREADS; ++i) {
            int q = tid + i * THREADS;
            if (q < BN * CPR) {
                int row = q / CPR, c = q % CPR;
                int kb = kt * BK + c * 8;
                bool ok = kb < ktot;
                const bf16* p = ok ? wt + (long long)(n0 + row) * ktot + kb : wt;
                cp_async16(smem_addr(sb + row * BK + ((c ^ swz<CPR>(row)) << 3)), p, ok);
            }
        }
    };

    float acc[MI][NI][4];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;

#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < ktiles) load_stage(s, s);
        cp_commit();
    }
    for (int kt = 0; kt < ktiles; ++kt) {
        cp_wait<STAGES - 2>();
        __syncthreads();
        const bf16* sa = sm + (kt % STAGES) * STAGE;
        const bf16* sb = sa + A_ELEMS;
#pragma unroll
        for (int kk = 0; kk < BK / 16; ++kk) {
            uint32_t af[MI][4];
#pragma unroll
            for (int i = 0; i < MI; ++i) {
                int row = wm0 + i * 16 + (lane & 15), c = kk * 2 + (lane >> 4);
                ldsm_x4(smem_addr(sa + row * BK + ((c ^ swz<CPR>(row)) << 3)), af[i]);
            }
#pragma unroll
            for (int jj = 0; jj < NI / 2; ++jj) {
                uint32_t bfr[4];
                int row = wn0 + jj * 16 + (lane & 7) + ((lane >> 4) << 3), c = kk * 2 + ((lane >> 3) & 1);
                ldsm_x4(smem_addr(sb + row * BK + ((c ^ swz<CPR>(row)) << 3)), bfr);
#pragma unroll
                for (int i = 0; i < MI; ++i) {
                    mma_bf16(acc[i][2 * jj], af[i], bfr[0], bfr[1]);
                    mma_bf16(acc[i][2 * jj + 1], af[i], bfr[2], bfr[3]);
                }
            }
        }
        int nk = kt + STAGES - 1;
        if (nk < ktiles) load_stage(nk % STAGES, nk);
        cp_commit();
    }
    cp_wait<0>();
    __syncthreads();

    // epilogue: bias + ReLU into a padded shared tile, then 16-byte rows to global (times the mask)
    constexpr int EP = BN + 8;
    bf16* se = sm;
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j) {
            int row = wm0 + i * 16 + (lane >> 2), col = wn0 + j * 8 + (lane & 3) * 2;
            float b0 = bias ? bias[n0 + col] : 0.f, b1 = bias ? bias[n0 + col + 1] : 0.f;
            float v0 = acc[i][j][0] + b0, v1 = acc[i][j][1] + b1, v2 = acc[i][j][2] + b0, v3 = acc[i][j][3] + b1;
            if (relu) {
                v0 = fmaxf(v0, 0.f); v1 = fmaxf(v1, 0.f); v2 = fmaxf(v2, 0.f); v3 = fmaxf(v3, 0.f);
            }
            *reinterpret_cast<__nv_bfloat162*>(se + row * EP + col) = __floats2bfloat162_rn(v0, v1);
            *reinterpret_cast<__nv_bfloat162*>(se + (row + 8) * EP + col) = __floats2bfloat162_rn(v2, v3);
        }
    __syncthreads();
    constexpr int CH = BN / 8;
    for (int q = tid; q < BM * CH; q += THREADS) {
        int row = q / CH, c = q % CH;
        long long v = m0 + row;
        if (v >= g.m) continue;
        uint4 val = *reinterpret_cast<const uint4*>(se + row * EP + c * 8);
        long long off = v * cout + n0 + c * 8;
        if (mask) {
            uint4 mk = *reinterpret_cast<const uint4*>(mask + off);
            uint32_t* pv = reinterpret_cast<uint32_t*>(&val);
            const uint32_t* pm = reinterpret_cast<const uint32_t*>(&mk);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                // keep each bf16 where the mask's bf16 is > 0 (sign bit clear and not +0)
                uint32_t lo = (pm[e] & 0xFFFFu), hi = pm[e] >> 16;
                uint32_t keep = ((lo & 0x8000u) == 0 && lo != 0 ? 0xFFFFu : 0u) |
                                ((hi & 0x8000u) == 0 && hi != 0 ? 0xFFFF0000u : 0u);
                pv[e] &= keep;
            }
        }
        *reinterpret_cast<uint4*>(y + off) = val;
    }
}

// ---------------------------------------------------------------------------------------------
// 3x3x3 convolution over a halo tile, for narrow outputs (BN = 16 or 32 channels): the CTA's 128
// output voxels are a 2 x 8 x 8 (z, y, x) block; for each 16-channel slice of the input it loads
// the 4 x 10 x 10 halo around that block once, and the slice's weights for all 27 taps, and forms
// every tap's A fragments by ldmatrix addressing into the halo (the 8 rows of one 8 x 8 matrix
// are 8 consecutive x of one line, i.e. 8 consecutive halo voxels).  The input is read once per
// tile instead of once per tap.  Halo and weight rows are 32 bytes (16 channels), their two
// 16-byte chunks swapped on every other group of 4 rows so the 8 rows of an ldmatrix phase fall
// in 8 different bank groups.
template <int BN>
__global__ void __launch_bounds__(128) conv3_halo_kernel(const bf16* __restrict__ x, const bf16* __restrict__ wt,
                                                         const float* __restrict__ bias,
                                                         const bf16* __restrict__ mask, bf16* __restrict__ y, Geo g,
                                                         int cin, int cout, int relu, int tiles_x, int tiles_y,
                                                         int tiles_z) {
    constexpr int TZ = 2, TY = 8, TX = 8, BM = TZ * TY * TX;
    constexpr int HZ = TZ + 2, HY = TY + 2, HX = TX + 2, HV = HZ * HY * HX;   // 400 halo voxels
    constexpr int WARPS_M = 4, WM = BM / WARPS_M, MI = WM / 16, NI = BN / 8;
    static_assert(NI % 2 == 0 && MI == 2, "tile shape");
    constexpr int ROWB = 32;                     // bytes per halo / weight row (16 channels)
    extern __shared__ __align__(1024) unsigned char dyn_smem[];
    unsigned char* sh = dyn_smem;                // [HV][32 B]
    unsigned char* sw = dyn_smem + HV * ROWB;    // [27][BN][32 B]

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm0 = warp * WM;
    int tile = blockIdx.x;
    const int txi = tile % tiles_x;
    tile /= tiles_x;
    const int tyi = tile % tiles_y;
    tile /= tiles_y;
    const int tzi = tile % tiles_z;
    const int n = tile / tiles_z;
    const int x0 = txi * TX, y0 = tyi * TY, z0 = tzi * TZ;
    const int n0 = blockIdx.y * BN;
    const long long vol0 = (long long)n * g.d * g.h * g.w;

    // halo-voxel index of this lane's A rows (tap offset added per tap)
    int hbase[MI];
#pragma unroll
    for (int i = 0; i < MI; ++i) {
        int r = wm0 + i * 16 + (lane & 15);
        int tx = r & 7, ty = (r >> 3) & 7, tz = r >> 6;
        hbase[i] = ((tz + 1) * HY + (ty + 1)) * HX + (tx + 1);
    }
    const int achunk = lane >> 4;                // A: lanes 16-31 read the second 8 channels

    float acc[MI][NI][4];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;

    const int slices = cin / 16;
    for (int sl = 0; sl < slices; ++sl) {
        const int c0 = sl * 16;
        // halo: HV rows x 2 chunks, zero outside the volume
        for (int q = tid; q < HV * 2; q += 128) {
            int hv = q >> 1, c = q & 1;
            int hx = hv % HX, hy = (hv / HX) % HY, hz = hv / (HX * HY);
            int zz = z0 + hz - 1, yy = y0 + hy - 1, xx = x0 + hx - 1;
            bool ok = zz >= 0 && zz < g.d && yy >= 0 && yy < g.h && xx >= 0 && xx < g.w;
            const bf16* p = ok ? x + (vol0 + ((long long)zz * g.h + yy) * g.w + xx) * cin + c0 + c * 8 : x;
            cp_async16(smem_addr(sh + hv * ROWB + ((c ^ ((hv >> 2) & 1)) << 4)), p, ok);
        }
        // weights of this slice for all taps: row (t, co), 16 channels
        for (int q = tid; q < 27 * BN * 2; q += 128) {
            int row = q >> 1, c = q & 1;
            int t = row / BN, co = row - t * BN;
            const bf16* p = wt + ((long long)(n0 + co) * 27 + t) * cin + c0 + c * 8;
            cp_async16(smem_addr(sw + row * ROWB + ((c ^ ((row >> 2) & 1)) << 4)), p, true);
        }
        cp_commit();
        cp_wait<0>();
        __syncthreads();
#pragma unroll 3
        for (int t = 0; t < 27; ++t) {
            const int off = (t / 9 - 1) * (HY * HX) + ((t / 3) % 3 - 1) * HX + (t % 3 - 1);
            uint32_t af[MI][4];
#pragma unroll
            for (int i = 0; i < MI; ++i) {
                int hv = hbase[i] + off;
                ldsm_x4(smem_addr(sh + hv * ROWB + ((achunk ^ ((hv >> 2) & 1)) << 4)), af[i]);
            }
#pragma unroll
            for (int jj = 0; jj < NI / 2; ++jj) {
                uint32_t bfr[4];
                int row = t * BN + jj * 16 + (lane & 7) + ((lane >> 4) << 3);
                int c = (lane >> 3) & 1;
                ldsm_x4(smem_addr(sw + row * ROWB + ((c ^ ((row >> 2) & 1)) << 4)), bfr);
#pragma unroll
                for (int i = 0; i < MI; ++i) {
                    mma_bf16(acc[i][2 * jj], af[i], bfr[0], bfr[1]);
                    mma_bf16(acc[i][2 * jj + 1], af[i], bfr[2], bfr[3]);
                }
            }
        }
        __syncthreads();                 // the next slice overwrites the halo and the weights
    }

    // epilogue: bias + ReLU into a padded shared tile, then 16-byte rows to global (times the mask)
    constexpr int EP = BN + 8;
    bf16* se = reinterpret_cast<bf16*>(dyn_smem);
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j) {
            int row = wm0 + i * 16 + (lane >> 2), col = j * 8 + (lane & 3) * 2;
            float b0 = bias ? bias[n0 + col] : 0.f, b1 = bias ? bias[n0 + col + 1] : 0.f;
            float v0 = acc[i][j][0] + b0, v1 = acc[i][j][1] + b1, v2 = acc[i][j][2] + b0, v3 = acc[i][j][3] + b1;
            if (relu) {
                v0 = fmaxf(v0, 0.f); v1 = fmaxf(v1, 0.f); v2 = fmaxf(v2, 0.f); v3 = fmaxf(v3, 0.f);
            }
            *reinterpret_cast<__nv_bfloat162*>(se + row * EP + col) = __floats2bfloat162_rn(v0, v1);
            *reinterpret_cast<__nv_bfloat162*>(se + (row + 8) * EP + col) = __floats2bfloat162_rn(v2, v3);
        }
    __syncthreads();
    constexpr int CH = BN / 8;
    for (int q = tid; q < BM * CH; q += 128) {
        int r = q / CH, c = q % CH;
        int xx = x0 + (r & 7), yy = y0 + ((r >> 3) & 7), zz = z0 + (r >> 6);
        if (xx >= g.w || yy >= g.h || zz >= g.d) continue;
        long long v = vol0 + ((long long)zz * g.h + yy) * g.w + xx;
        uint4 val = *reinterpret_cast<const uint4*>(se + r * EP + c * 8);
        long long o = v * cout + n0 + c * 8;
        if (mask) {
            uint4 mk = *reinterpret_cast<const uint4*>(mask + o);
            uint32_t* pv = reinterpret_cast<uint32_t*>(&val);
            const uint32_t* pm = reinterpret_cast<const uint32_t*>(&mk);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                uint32_t lo = (pm[e] & 0xFFFFu), hi = pm[e] >> 16;
                uint32_t keep = ((lo & 0x8000u) == 0 && lo != 0 ? 0xFFFFu : 0u) |
                                ((hi & 0x8000u) == 0 && hi != 0 ? 0xFFFF0000u : 0u);
                pv[e] &= keep;
            }
        }
        *reinterpret_cast<uint4*>(y + o) = val;
    }
}

// ---------------------------------------------------------------------------------------------
// Fifth-generation tensor cores (tcgen05): descriptors, bounded waits, tensor-memory loads.  A wait
// that gives up sets g_dn_fault, which mcxg_dn_check reports.
__device__ unsigned g_dn_fault;

// kind::f16 instruction descriptor: FP32 accumulator, BF16 A and B, both K-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

// Waits for the completion of the mbarrier phase of parity `parity`; false after about a second.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    const long long t0 = clock64();
    while (true) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        if (clock64() - t0 > 2000000000LL) return false;
    }
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

// A kernel launched by launch_chained may start while the one before it on the stream still runs: it touches nothing but its
// own shared and tensor memory until chain_wait, which returns once that one has finished and its writes are seen.
// Every thread calls it, so that a kernel's end means the end of all before it.  chain_next lets the next such
// kernel start as this one's CTAs leave.
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
#include "conv3_roll.cuh"
#include "conv3_stream.cuh"
#include "conv3_wgrad.cuh"

// ---------------------------------------------------------------------------------------------
// Weight gradient: dW[co, n] += sum_v dY[v, co] * X[v + off(t), ci], n = t*Cin + ci, over the
// voxel slice [blockIdx.y*kslice, +kslice).  BM = Cout (the whole output-channel range), BN = 64
// columns of (tap, ci); 128 threads; K staged 32 voxels at a time.
template <int BM, int STAGES>
__global__ void __launch_bounds__(128) conv_wgrad_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x,
                                                         float* __restrict__ dw, Geo g, int cin, int taps,
                                                         long long kslice) {
    constexpr int BN = 64, BK = 32;
    constexpr int CPA = BM / 8, CPB = BN / 8;
    constexpr int WARPS_M = BM >= 32 ? 2 : 1;
    constexpr int WARPS_N = 4 / WARPS_M;
    constexpr int WM = BM / WARPS_M, WN = BN / WARPS_N;
    constexpr int MI = WM / 16, NI = WN / 8;
    constexpr int A_ELEMS = BK * BM, B_ELEMS = BK * BN;
    constexpr int STAGE = A_ELEMS + B_ELEMS;
    static_assert(NI % 2 == 0 && MI >= 1, "tile shape");

    extern __shared__ __align__(1024) unsigned char dyn_smem[];
    bf16* sm = reinterpret_cast<bf16*>(dyn_smem);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm0 = (warp / WARPS_N) * WM, wn0 = (warp % WARPS_N) * WN;
    const int ntot = taps * cin;
    const int nt0 = blockIdx.x * BN;
    const long long kbeg = (long long)blockIdx.y * kslice;
    const long long kend = min(g.m, kbeg + kslice);
    if (kbeg >= kend) return;
    const int ktiles = (int)((kend - kbeg + BK - 1) / BK);
    const long long vvol = (long long)g.d * g.h * g.w;

    // the B (input) chunks this thread loads: one fixed column chunk (tap, 8 channels) and rows
    // tid / CPB + 16 i, whose voxel coordinates advance by BK voxels per stage (stages are
    // loaded in order), so no division runs inside the K loop
    constexpr int B_IT = BK * CPB / 128;
    static_assert(B_IT * 128 == BK * CPB && 128 % CPB == 0, "B loader shape");
    const int bc = tid % CPB;
    const int ncol = nt0 + bc * 8;
    const bool col_ok = ncol < ntot;
    const int tap = col_ok ? ncol / cin : 0, ci = col_ok ? ncol - tap * cin : 0;
    int tz = 0, ty = 0, tx = 0;
    if (taps == 27) {
        tz = tap / 9 - 1;
        ty = (tap / 3) % 3 - 1;
        tx = tap % 3 - 1;
    }
    const long long delta = (long long)tz * g.h * g.w + ty * g.w + tx;
    long long bv[B_IT];
    int bz[B_IT], by[B_IT], bx[B_IT];
#pragma unroll
    for (int i = 0; i < B_IT; ++i) {
        bv[i] = kbeg + tid / CPB + i * (128 / CPB);
        long long r = bv[i] % vvol;
        bx[i] = (int)(r % g.w);
        by[i] = (int)((r / g.w) % g.h);
        bz[i] = (int)(r / ((long long)g.w * g.h));
    }

    auto load_stage = [&](int stage, int kt) {
        bf16* sa = sm + stage * STAGE;
        bf16* sb = sa + A_ELEMS;
        const long long vb = kbeg + (long long)kt * BK;
        for (int q = tid; q < BK * CPA; q += 128) {
            int row = q / CPA, c = q % CPA;
            long long v = vb + row;
            bool ok = v < kend;
            const bf16* p = ok ? dy + v * BM + c * 8 : dy;
            cp_async16(smem_addr(sa + row * BM + ((c ^ swz<CPA>(row)) << 3)), p, ok);
        }
#pragma unroll
        for (int i = 0; i < B_IT; ++i) {
            int row = tid / CPB + i * (128 / CPB);
            int zz = bz[i] + tz, yy = by[i] + ty, xx = bx[i] + tx;
            bool ok = col_ok && bv[i] < kend && zz >= 0 && zz < g.d && yy >= 0 && yy < g.h && xx >= 0 && xx < g.w;
            const bf16* p = ok ? x + (bv[i] + delta) * cin + ci : x;
            cp_async16(smem_addr(sb + row * BN + ((bc ^ swz<CPB>(row)) << 3)), p, ok);
            // next stage: BK voxels further on
            bv[i] += BK;
            bx[i] += BK;
            while (bx[i] >= g.w) {
                bx[i] -= g.w;
                if (++by[i] >= g.h) {
                    by[i] = 0;
                    if (++bz[i] >= g.d) bz[i] = 0;
                }
            }
        }
    };

    float acc[MI][NI][4];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;

#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < ktiles) load_stage(s, s);
        cp_commit();
    }
    for (int kt = 0; kt < ktiles; ++kt) {
        cp_wait<STAGES - 2>();
        __syncthreads();
        const bf16* sa = sm + (kt % STAGES) * STAGE;
        const bf16* sb = sa + A_ELEMS;
#pragma unroll
        for (int kk = 0; kk < BK / 16; ++kk) {
            const int qm = lane >> 3, r8 = lane & 7;
            uint32_t af[MI][4];
#pragma unroll
            for (int i = 0; i < MI; ++i) {
                int row = kk * 16 + r8 + ((qm >> 1) << 3);
                int c = (wm0 + i * 16) / 8 + (qm & 1);
                ldsm_x4_t(smem_addr(sa + row * BM + ((c ^ swz<CPA>(row)) << 3)), af[i]);
            }
#pragma unroll
            for (int jj = 0; jj < NI / 2; ++jj) {
                uint32_t bfr[4];
                int row = kk * 16 + r8 + ((qm & 1) << 3);
                int c = (wn0 + jj * 16) / 8 + (qm >> 1);
                ldsm_x4_t(smem_addr(sb + row * BN + ((c ^ swz<CPB>(row)) << 3)), bfr);
#pragma unroll
                for (int i = 0; i < MI; ++i) {
                    mma_bf16(acc[i][2 * jj], af[i], bfr[0], bfr[1]);
                    mma_bf16(acc[i][2 * jj + 1], af[i], bfr[2], bfr[3]);
                }
            }
        }
        int nk = kt + STAGES - 1;
        if (nk < ktiles) load_stage(nk % STAGES, nk);
        cp_commit();
    }
    cp_wait<0>();

#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j) {
            int co = wm0 + i * 16 + (lane >> 2);
            int n = nt0 + wn0 + j * 8 + (lane & 3) * 2;
            if (n < ntot) {
                atomicAdd(dw + (long long)co * ntot + n, acc[i][j][0]);
                atomicAdd(dw + (long long)(co + 8) * ntot + n, acc[i][j][2]);
            }
            if (n + 1 < ntot) {
                atomicAdd(dw + (long long)co * ntot + n + 1, acc[i][j][1]);
                atomicAdd(dw + (long long)(co + 8) * ntot + n + 1, acc[i][j][3]);
            }
        }
}

// db[c] += sum_v dY[v, c]
__global__ void bias_grad_kernel(const bf16* __restrict__ dy, float* __restrict__ db, long long m, int c,
                                 long long rows_per_block) {
    const int lanes = blockDim.x / c;  // rows processed side by side
    const int ch = threadIdx.x % c, r0 = threadIdx.x / c;
    long long beg = blockIdx.x * rows_per_block, end = min(m, beg + rows_per_block);
    float s = 0.f;
    for (long long v = beg + r0; v < end; v += lanes) s += __bfloat162float(dy[v * c + ch]);
    atomicAdd(db + ch, s);
}

__device__ __forceinline__ void load8(const bf16* p, float (&f)[8]) {
    uint4 u = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        float2 t = __bfloat1622float2(h[e]);
        f[2 * e] = t.x;
        f[2 * e + 1] = t.y;
    }
}
__device__ __forceinline__ void store8(bf16* p, const float (&f)[8]) {
    uint4 u;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
    for (int e = 0; e < 4; ++e) h[e] = __floats2bfloat162_rn(f[2 * e], f[2 * e + 1]);
    *reinterpret_cast<uint4*>(p) = u;
}

// The same for channels in whole 16-byte chunks: a thread keeps one chunk of 8 channels and walks rows a grid apart, four in
// flight, the block adds its rows by shuffles and through shared memory, one atomic a channel and block.  Bound by the read of
// dY and a launch: 524288 rows of 16 channels (17 MB) took 18.7 us with 2-byte loads, one channel a thread and 128 blocks,
// 6.3 with a row in flight and a thread adding a channel's 128 partial sums, and take 4.3.
__global__ void __launch_bounds__(256) bias_grad8_kernel(const bf16* dy, float* db, long long m, int c) {
    chain_next();
    chain_wait();
    __shared__ float part[8][256];
    const int cc = c / 8, rows = 256 / cc;
    const int ch = threadIdx.x % cc, r0 = threadIdx.x / cc;
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const long long step = (long long)gridDim.x * rows;
    for (long long v = (long long)blockIdx.x * rows + r0; v < m; v += 4 * step) {
        float f[4][8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {           // four rows in flight
            if (v + i * step < m) {
                load8(dy + (v + i * step) * c + ch * 8, f[i]);
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) f[i][e] = 0.f;
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int e = 0; e < 8; ++e) s[e] += f[i][e];
    }
    // over the warp's lanes of one chunk (cc is a power of two of at most 32), then over the warps
    for (int o = cc; o < 32; o *= 2)
#pragma unroll
        for (int e = 0; e < 8; ++e) s[e] += __shfl_xor_sync(0xffffffffu, s[e], o);
    if ((int)(threadIdx.x & 31) < cc) {
#pragma unroll
        for (int e = 0; e < 8; ++e) part[threadIdx.x / 32][ch * 8 + e] = s[e];
    }
    __syncthreads();
    if ((int)threadIdx.x < c) {
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += part[w][threadIdx.x];
        atomicAdd(db + threadIdx.x, t);
    }
}

// 2x2x2 average pooling; (d, h, w) are the fine grid's sizes.  One thread per coarse voxel and
// 8-channel chunk.
__global__ void pool_kernel(const bf16* x, bf16* y, int nvol, int d, int h, int w, int c) {
    chain_next();
    chain_wait();
    const int d2 = d / 2, h2 = h / 2, w2 = w / 2, cc = c / 8;
    long long total = (long long)nvol * d2 * h2 * w2 * cc;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total; q += (long long)gridDim.x * blockDim.x) {
        int ch = (int)(q % cc);
        long long v = q / cc;
        int xx = (int)(v % w2), yy = (int)((v / w2) % h2), zz = (int)((v / ((long long)w2 * h2)) % d2);
        long long n = v / ((long long)w2 * h2 * d2);
        float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int k = 0; k < 8; ++k) {
            long long fv = ((n * d + 2 * zz + (k >> 2)) * h + 2 * yy + ((k >> 1) & 1)) * w + 2 * xx + (k & 1);
            float f[8];
            load8(x + fv * c + ch * 8, f);
#pragma unroll
            for (int e = 0; e < 8; ++e) s[e] += f[e];
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) s[e] *= 0.125f;
        store8(y + v * c + ch * 8, s);
    }
}

// q / d for q < 2^31 by a multiplication: s = ceil(log2 d), m = floor(2^32 (2^s - d) / d) + 1, q / d = (hi(q m) + q) >> s
// (Granlund and Montgomery, "Division by invariant integers using multiplication", 1994).
struct FastDiv {
    unsigned d, m, s;
    explicit FastDiv(unsigned div) : d(div), m(0), s(0) {
        while ((1ull << s) < d) ++s;
        m = (unsigned)((((1ull << s) - d) << 32) / d + 1);
    }
    __device__ __forceinline__ unsigned div(unsigned q) const { return (__umulhi(q, m) + q) >> s; }
};

// cat[v, 0:c1] = low[parent(v)], cat[v, c1:c1+c2] = skip[v]; (d, h, w) fine sizes.  A thread moves four 16-byte chunks a
// block apart, all four read before the first is written, their places found with 32-bit multiplications.  Bound by the
// write: 128^3 of 32 + 16 channels (84 MB read, 201 MB written) in 43 us, 6.6 TB/s (a chunk
// at a time, 64-bit divisions: 98).
__global__ void __launch_bounds__(256) upcat4_kernel(const uint4* low, const uint4* skip, uint4* cat, unsigned total,
                                                     unsigned k1, FastDiv ct, FastDiv w, FastDiv h, FastDiv d) {
    const unsigned q0 = blockIdx.x * 1024u + threadIdx.x, k2 = ct.d - k1;
    chain_next();
    chain_wait();
    uint4 u[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const unsigned q = q0 + i * 256u;
        if (q >= total) break;
        const unsigned v = ct.div(q), ch = q - v * ct.d;
        if (ch < k1) {
            const unsigned yz = w.div(v), x = v - yz * w.d, zn = h.div(yz), y = yz - zn * h.d, n = d.div(zn), z = zn - n * d.d;
            const unsigned pv = ((n * (d.d >> 1) + (z >> 1)) * (h.d >> 1) + (y >> 1)) * (w.d >> 1) + (x >> 1);
            u[i] = low[(size_t)pv * k1 + ch];
        } else {
            u[i] = skip[(size_t)v * k2 + (ch - k1)];
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (q0 + i * 256u < total) cat[q0 + i * 256u] = u[i];
}

// The same for 2^31 chunks and more.
__global__ void upcat_kernel(const bf16* __restrict__ low, const bf16* __restrict__ skip, bf16* __restrict__ cat,
                             int nvol, int d, int h, int w, int c1, int c2) {
    const int ct = (c1 + c2) / 8;
    long long total = (long long)nvol * d * h * w * ct;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total; q += (long long)gridDim.x * blockDim.x) {
        int ch = (int)(q % ct);
        long long v = q / ct;
        const bf16* src;
        if (ch * 8 < c1) {
            int xx = (int)(v % w), yy = (int)((v / w) % h), zz = (int)((v / ((long long)w * h)) % d);
            long long n = v / ((long long)w * h * d);
            long long pv = ((n * (d / 2) + zz / 2) * (h / 2) + yy / 2) * (w / 2) + xx / 2;
            src = low + pv * c1 + ch * 8;
        } else {
            src = skip + v * c2 + (ch * 8 - c1);
        }
        *reinterpret_cast<uint4*>(cat + v * (c1 + c2) + ch * 8) = *reinterpret_cast<const uint4*>(src);
    }
}

// dlow[u, c] = (sum over the 8 children of dcat[child, c]) * (low[u, c] > 0), c < c1.
__global__ void upcat_bwd_kernel(const bf16* __restrict__ dcat, const bf16* __restrict__ low, bf16* __restrict__ dlow,
                                 int nvol, int d, int h, int w, int c1, int c2) {
    const int d2 = d / 2, h2 = h / 2, w2 = w / 2, cc = c1 / 8, ct = c1 + c2;
    long long total = (long long)nvol * d2 * h2 * w2 * cc;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total; q += (long long)gridDim.x * blockDim.x) {
        int ch = (int)(q % cc);
        long long u = q / cc;
        int xx = (int)(u % w2), yy = (int)((u / w2) % h2), zz = (int)((u / ((long long)w2 * h2)) % d2);
        long long n = u / ((long long)w2 * h2 * d2);
        float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int k = 0; k < 8; ++k) {
            long long fv = ((n * d + 2 * zz + (k >> 2)) * h + 2 * yy + ((k >> 1) & 1)) * w + 2 * xx + (k & 1);
            float f[8];
            load8(dcat + fv * ct + ch * 8, f);
#pragma unroll
            for (int e = 0; e < 8; ++e) s[e] += f[e];
        }
        float lv[8];
        load8(low + u * c1 + ch * 8, lv);
#pragma unroll
        for (int e = 0; e < 8; ++e) s[e] = lv[e] > 0.f ? s[e] : 0.f;
        store8(dlow + u * c1 + ch * 8, s);
    }
}

// denc[v, c] = (dpool[parent(v), c] / 8 + dcat[v, c1 + c]) * (enc[v, c] > 0); dcat may be null
// (no skip path).  (d, h, w) fine sizes; c = encoder channels.
__global__ void unpool_add_kernel(const bf16* __restrict__ dpool, const bf16* __restrict__ dcat,
                                  const bf16* __restrict__ enc, bf16* __restrict__ denc, int nvol, int d, int h, int w,
                                  int c1, int c) {
    const int cc = c / 8;
    long long total = (long long)nvol * d * h * w * cc;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total; q += (long long)gridDim.x * blockDim.x) {
        int ch = (int)(q % cc);
        long long v = q / cc;
        int xx = (int)(v % w), yy = (int)((v / w) % h), zz = (int)((v / ((long long)w * h)) % d);
        long long n = v / ((long long)w * h * d);
        long long pv = ((n * (d / 2) + zz / 2) * (h / 2) + yy / 2) * (w / 2) + xx / 2;
        float a[8], b[8], e8[8];
        load8(dpool + pv * c + ch * 8, a);
        if (dcat) load8(dcat + v * (c1 + c) + c1 + ch * 8, b);
        else
            for (int e = 0; e < 8; ++e) b[e] = 0.f;
        load8(enc + v * c + ch * 8, e8);
        float o[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = e8[e] > 0.f ? a[e] * 0.125f + b[e] : 0.f;
        store8(denc + v * c + ch * 8, o);
    }
}

// Head: out[v] = xres[v] + b + sum_c w[c] * act[v, c] (16 channels).  With a target, also the
// masked L1 loss, dact = g * w * (act > 0), dw += g * act, db += g, g = sign(out - t) * valid * inv.
__global__ void __launch_bounds__(256) head_kernel(const bf16* act, const float* xres, const float* w, const float* b,
                                                   const float* target, const float* valid, float* out, bf16* dact, float* dw,
                                                   float* db, float* loss, long long m, float inv) {
    __shared__ float red[8][18];
    chain_next();
    chain_wait();
    float gw[16], gb = 0.f, ls = 0.f;
#pragma unroll
    for (int c = 0; c < 16; ++c) gw[c] = 0.f;
    float wc[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) wc[c] = w[c];
    const float bias = b[0];
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < m; v += (long long)gridDim.x * blockDim.x) {
        float a[16];
        float lo[8], hi[8];
        load8(act + v * 16, lo);
        load8(act + v * 16 + 8, hi);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            a[e] = lo[e];
            a[8 + e] = hi[e];
        }
        float o = xres[v] + bias;
#pragma unroll
        for (int c = 0; c < 16; ++c) o = fmaf(wc[c], a[c], o);
        if (out) out[v] = o;
        if (target) {
            float diff = o - target[v], vl = valid[v];
            ls += fabsf(diff) * vl;
            float gr = (diff > 0.f ? 1.f : (diff < 0.f ? -1.f : 0.f)) * vl * inv;
            gb += gr;
#pragma unroll
            for (int c = 0; c < 16; ++c) gw[c] += gr * a[c];
            float da[16];
#pragma unroll
            for (int c = 0; c < 16; ++c) da[c] = a[c] > 0.f ? gr * wc[c] : 0.f;
            float d0[8], d1[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                d0[e] = da[e];
                d1[e] = da[8 + e];
            }
            store8(dact + v * 16, d0);
            store8(dact + v * 16 + 8, d1);
        }
    }
    if (!target) return;
    // block reduction of the 18 sums (16 weights, bias, loss)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float vals[18];
#pragma unroll
    for (int c = 0; c < 16; ++c) vals[c] = gw[c];
    vals[16] = gb;
    vals[17] = ls;
#pragma unroll
    for (int k = 0; k < 18; ++k) {
        float s = vals[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) red[warp][k] = s;
    }
    __syncthreads();
    if (threadIdx.x < 18) {
        float s = 0.f;
        for (int k = 0; k < (int)(blockDim.x / 32); ++k) s += red[k][threadIdx.x];
        if (threadIdx.x < 16) atomicAdd(dw + threadIdx.x, s);
        else if (threadIdx.x == 16) atomicAdd(db, s);
        else atomicAdd(loss, s);
    }
}

// Input features of one voxel (16 channels, 0..6 used), with l0, l3, l5 = log10(m + 1e-10) of the
// noisy fluence F and of its means over the in-bounds voxels of the 3x3x3 and 5x5x5
// neighbourhoods:
//   0: (l3 + 5) / 3      1: clamp(4 (l0 - l3), -4, 4)      2: clamp(4 (l5 - l3), -4, 4)
//   3: 1 where F is 0    4: log10(mua) + 2    5: log10(mus (1 - g))    6: (log10(photons) - 5.5) * 2
// and xres[v] = l3, the residual base the head adds its correction to.  The means are taken in
// linear fluence, where a voxel no photon reached is a zero among its neighbours rather than a
// -10 outlier as in log space; channels 1 and 2 hand the network the noise and the curvature at
// the scale of its correction instead of as small differences of large inputs.
//
// A block covers 4 TX x (128 / TX) x 4 voxels from a shared-memory copy of them with a halo of two (outside the volume
// zeros, which add nothing), a thread four neighbours in x, whose windows share the eight values it reads a row: 75 shared
// loads for 500 additions, each voxel's sum in the order z, y, x.  The copy's loads are all issued before any is
// used (one after another: 60 us), the media's two channels come from a table by label.  128^3: 38 us, 64^3 7.4 (125
// bounds-checked global loads a voxel: 139 and 23); 67 of its 86 MB are x0, the rest of the time is arithmetic.
template <int TX>
__global__ void __launch_bounds__(512) pack_kernel(const float* __restrict__ flux, const uint8_t* __restrict__ label,
                                                   const float* __restrict__ props, const float* __restrict__ log_photons,
                                                   bf16* __restrict__ x0, float* __restrict__ xres, Geo g, int nprop,
                                                   int tiles_x, int tiles_y, int tiles_z, long long tiles, int wide,
                                                   int vec) {
    constexpr int X = 4 * TX, Y = 128 / TX, Z = 4, W = X + 8;          // the copy starts four voxels left of the tile
    __shared__ __align__(16) float s_f[Z + 4][Y + 4][W];
    __shared__ uint32_t s_media[256];
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX % Y, tz = threadIdx.x / 128;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const long long vvol = (long long)g.d * g.h * g.w;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
        long long r = t;
        const int x0t = (int)(r % tiles_x) * X;
        r /= tiles_x;
        const int y0t = (int)(r % tiles_y) * Y;
        r /= tiles_y;
        const int z0t = (int)(r % tiles_z) * Z, n = (int)(r / tiles_z);
        const float* fl = flux + n * vvol;
        // the copy: a warp a row, all of its rows' loads in flight before the first is stored
        constexpr int ROWS = (Z + 4) * (Y + 4), PER = (ROWS + 15) / 16, COLS = (W + 31) / 32;
        float v0[PER][COLS];
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int row = warp + 16 * i, yy = y0t - 2 + row % (Y + 4), zz = z0t - 2 + row / (Y + 4);
            const bool in = (unsigned)yy < (unsigned)g.h && (unsigned)zz < (unsigned)g.d && row < ROWS;
            const float* src = fl + ((long long)zz * g.h + yy) * g.w;
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                const int xx = x0t - 4 + lane + 32 * c;
                v0[i][c] = in && (unsigned)xx < (unsigned)g.w ? src[xx] : 0.f;
            }
        }
        // channels 4 and 5 by label
        for (int i = threadIdx.x; i < min(nprop, 256); i += 512) {
            const float* pr = props + ((long long)n * nprop + i) * 4;
            const float f4 = pr[0] > 0.f ? log10f(pr[0]) + 2.f : -2.f, musp = pr[1] * (1.f - pr[2]);
            const __nv_bfloat162 h2 = __floats2bfloat162_rn(f4, musp > 0.f ? log10f(musp) : -3.f);
            s_media[i] = *reinterpret_cast<const uint32_t*>(&h2);
        }
#pragma unroll
        for (int i = 0; i < PER; ++i)
#pragma unroll
            for (int c = 0; c < COLS; ++c)
                if (warp + 16 * i < ROWS && lane + 32 * c < W)
                    (&s_f[0][0][0])[(warp + 16 * i) * W + lane + 32 * c] = fmaxf(v0[i][c], 0.f);
        __syncthreads();
        float s3[4] = {0.f, 0.f, 0.f, 0.f}, s5[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int dz = 0; dz < 5; ++dz)
#pragma unroll
            for (int dy = 0; dy < 5; ++dy) {
                const float* row = &s_f[tz + dz][ty + dy][4 * tx];
                const float2 a = *reinterpret_cast<const float2*>(row + 2), c = *reinterpret_cast<const float2*>(row + 8);
                const float4 b = *reinterpret_cast<const float4*>(row + 4);
                const float v[8] = {a.x, a.y, b.x, b.y, b.z, b.w, c.x, c.y};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
#pragma unroll
                    for (int dx = 0; dx < 5; ++dx) s5[j] += v[j + dx];
                    if (dz >= 1 && dz <= 3 && dy >= 1 && dy <= 3) {
#pragma unroll
                        for (int dx = 1; dx < 4; ++dx) s3[j] += v[j + dx];
                    }
                }
            }
        const int y = y0t + ty, z = z0t + tz;
        if (y < g.h && z < g.d) {
            auto within = [](int p, int reach, int size) { return min(p + reach, size - 1) - max(p - reach, 0) + 1; };
            const int c3yz = within(y, 1, g.h) * within(z, 1, g.d), c5yz = within(y, 2, g.h) * within(z, 2, g.d);
            const int x1 = x0t + 4 * tx;
            const long long v1 = n * vvol + ((long long)z * g.h + y) * g.w + x1;
            float fv[4], res[4];
            int lab[4];
            if (vec) {
                if (x1 < g.w) {
                    const float4 a = *reinterpret_cast<const float4*>(flux + v1);
                    const uchar4 b = *reinterpret_cast<const uchar4*>(label + v1);
                    fv[0] = a.x, fv[1] = a.y, fv[2] = a.z, fv[3] = a.w;
                    lab[0] = b.x, lab[1] = b.y, lab[2] = b.z, lab[3] = b.w;
                }
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (x1 + j < g.w) fv[j] = flux[v1 + j], lab[j] = label[v1 + j];
            }
            const float code = (log_photons[n] - 5.5f) * 2.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int x = x1 + j;
                if (x >= g.w) break;
                const long long v = v1 + j;
                const int c3 = c3yz * within(x, 1, g.w), c5 = c5yz * within(x, 2, g.w);
                float l0 = log10f(fmaxf(fv[j], 0.f) + 1e-10f);
                float l3 = log10f(s3[j] / (float)c3 + 1e-10f);
                float l5 = log10f(s5[j] / (float)c5 + 1e-10f);
                const __nv_bfloat162 h[3] = {
                    __floats2bfloat162_rn((l3 + 5.f) * (1.f / 3.f), fminf(fmaxf(4.f * (l0 - l3), -4.f), 4.f)),
                    __floats2bfloat162_rn(fminf(fmaxf(4.f * (l5 - l3), -4.f), 4.f), fv[j] <= 0.f ? 1.f : 0.f),
                    __floats2bfloat162_rn(code, 0.f)};
                const uint32_t* u = reinterpret_cast<const uint32_t*>(h);
                const uint32_t media = s_media[min(lab[j], nprop - 1)];
                bf16* o = x0 + v * 16;
                if (wide) {         // a voxel's 32 bytes at once
                    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %5, %5, %5};\n" ::"l"(o), "r"(u[0]), "r"(u[1]),
                                 "r"(media), "r"(u[2]), "r"(0u)
                                 : "memory");
                } else {
                    reinterpret_cast<uint4*>(o)[0] = make_uint4(u[0], u[1], media, u[2]);
                    reinterpret_cast<uint4*>(o)[1] = make_uint4(0u, 0u, 0u, 0u);
                }
                res[j] = l3;
                if (!vec) xres[v] = l3;
            }
            if (vec && x1 < g.w) *reinterpret_cast<float4*>(xres + v1) = make_float4(res[0], res[1], res[2], res[3]);
        }
        __syncthreads();
    }
}

// AdamW on fp32 master weights (decoupled weight decay), gradient cleared after use.  Writes the
// bf16 weights and, for a convolution (taps > 0), the flipped transposed copy the data gradient
// runs on: wt[ci][taps-1-t][co] = w[co][t][ci].
__global__ void adamw_kernel(float* __restrict__ master, float* __restrict__ grad, float* __restrict__ m1,
                             float* __restrict__ m2, bf16* __restrict__ w16, bf16* __restrict__ wt16, long long n,
                             int cout, int taps, int cin, float lr, float b1, float b2, float eps, float wd,
                             float bc1, float bc2) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float gr = grad[i];
        float a = b1 * m1[i] + (1.f - b1) * gr;
        float s = b2 * m2[i] + (1.f - b2) * gr * gr;
        m1[i] = a;
        m2[i] = s;
        float p = master[i];
        p -= lr * (wd * p + (a / bc1) / (sqrtf(s / bc2) + eps));
        master[i] = p;
        grad[i] = 0.f;
        bf16 pb = __float2bfloat16_rn(p);
        if (w16) w16[i] = pb;
        if (wt16 && taps > 0) {
            int ci = (int)(i % cin);
            int t = (int)((i / cin) % taps);
            int co = (int)(i / ((long long)cin * taps));
            wt16[((long long)ci * taps + (taps - 1 - t)) * cout + co] = pb;
        }
    }
}

thread_local char g_err[256];

int fail(const char* msg) {
    snprintf(g_err, sizeof(g_err), "%s", msg);
    return -1;
}

int launched() {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        snprintf(g_err, sizeof(g_err), "denoiser kernel launch: %s", cudaGetErrorString(e));
        return -(int)e;
    }
    return 0;
}

// A launch that may overlap the end of the kernel before it on the stream (chain_wait in the kernel holds it back).  The
// network is two dozen kernels of 5 to 120 us: their launches, barriers and tensor memory set up behind the one before took
// a 128^3 forward pass from 633 to 585 us, a convolution in a row of its kind from 46.3 to 42.5 (16 to 16 at 128^3).
template <class... P, class... A>
int launch_chained(void (*kern)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
    return launched();
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int grid_for(long long work, int block) {
    long long g = (work + block - 1) / block;
    return (int)(g < 1 ? 1 : (g > 152 * 32 ? 152 * 32 : g));
}

template <int BM, int BN, int BK, int WARPS_M, int WARPS_N, int STAGES>
int conv_fwd_launch(const bf16* x, const bf16* w, const float* bias, const bf16* mask, bf16* y, Geo g, int cin,
                    int cout, int taps, int relu, cudaStream_t st) {
    constexpr int stage_bytes = (BM + BN) * BK * 2;
    constexpr int epi_bytes = BM * (BN + 8) * 2;
    constexpr int smem = STAGES * stage_bytes > epi_bytes ? STAGES * stage_bytes : epi_bytes;
    auto kern = conv_fwd_kernel<BM, BN, BK, WARPS_M, WARPS_N, STAGES>;
    static bool attr = false;
    if (!attr) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        attr = true;
    }
    dim3 grid((unsigned)((g.m + BM - 1) / BM), (unsigned)(cout / BN));
    kern<<<grid, 32 * WARPS_M * WARPS_N, smem, st>>>(x, w, bias, mask, y, g, cin, cout, taps, relu);
    return launched();
}

// Tile per output width: 128 voxels x (128 | 64 | 32 | 16) channels; narrow outputs take deeper
// K stages and fewer, taller warp tiles (two 16-row fragments per warp) so that each B fragment
// feeds more MMAs.
template <int BN>
int conv3_halo_launch(const bf16* x, const bf16* w, const float* bias, const bf16* mask, bf16* y, Geo g, int cin,
                      int cout, int relu, cudaStream_t st) {
    constexpr int smem_in = 400 * 32 + 27 * BN * 32;
    constexpr int smem_epi = 128 * (BN + 8) * 2;
    constexpr int smem = smem_in > smem_epi ? smem_in : smem_epi;
    auto kern = conv3_halo_kernel<BN>;
    static bool attr = false;
    if (!attr) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        attr = true;
    }
    const int tx = (g.w + 7) / 8, ty = (g.h + 7) / 8, tz = (g.d + 1) / 2;
    const long long tiles = (long long)g.nvol * tx * ty * tz;
    if (tiles >= (1LL << 31)) return fail("conv: too many tiles");
    kern<<<dim3((unsigned)tiles, (unsigned)(cout / BN)), 128, smem, st>>>(x, w, bias, mask, y, g, cin, cout, relu, tx, ty,
                                                                          tz);
    return launched();
}

// cuTensorMapEncodeTiled, found through the runtime (the engine links no driver library)
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
    }
    return fn;
}

// Shared memory of conv3_roll_kernel beside its barriers.
constexpr int kRollSmem = 225 * 1024;

// Lets a kernel have all of kRollSmem, once per device (`done`: a bit each, the kernel's own); asking at every launch cost
// the small layers, which take 8 us of host time a call, half a microsecond.
template <class K>
void allow_smem(K kern, int dev, std::atomic<unsigned long long>& done) {
    const unsigned long long bit = dev >= 0 && dev < 64 ? 1ull << dev : 0ull;
    if (bit && (done.load(std::memory_order_relaxed) & bit)) return;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kRollSmem) == cudaSuccess)
        done.fetch_or(bit, std::memory_order_relaxed);
}

// Launch of conv3_roll_kernel for BN output channels a block (BN divides cout).  Returns 1 where its planes are too many to
// count in 32 bits (volumes of a voxel a plane, many channel blocks): the general kernels count voxels.
template <int BN, bool TAPS>
int conv3_roll_launch(const bf16* x, const bf16* w, const float* bias, const bf16* mask, bf16* y, Geo g, int cin,
                      int cout, int relu, int dev, int sms, cudaStream_t st) {
    using S = RollShape<BN>;
    auto encode = tensor_map_encoder();
    if (!encode) return fail("conv: cuTensorMapEncodeTiled is not available");
    CUtensorMap xmap, wmap;
    {
        // activations [nvol][d][h][w][cin], a box of 16 channels of two halo planes (one in tap-major order)
        const cuuint64_t dims[5] = {(cuuint64_t)cin, (cuuint64_t)g.w, (cuuint64_t)g.h, (cuuint64_t)g.d, (cuuint64_t)g.nvol};
        const cuuint64_t strides[4] = {(cuuint64_t)cin * 2, (cuuint64_t)g.w * cin * 2, (cuuint64_t)g.h * g.w * cin * 2,
                                       (cuuint64_t)g.d * g.h * g.w * cin * 2};
        const cuuint32_t box[5] = {16, (cuuint32_t)S::HX, (cuuint32_t)S::HY, TAPS ? 1u : 2u, 1};
        const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
        if (encode(&xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<bf16*>(x), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return fail("conv: cuTensorMapEncodeTiled rejected the activation layout");
    }
    {
        // weights [cout][dz][dydx][cin] seen as (ci, co, dz, dydx): a box of a slice lands as the rows
        // (dydx, dz, co) that the MMAs of N = 3 BN read
        const cuuint64_t dims[4] = {(cuuint64_t)cin, (cuuint64_t)cout, 3, 9};
        const cuuint64_t strides[3] = {(cuuint64_t)27 * cin * 2, (cuuint64_t)9 * cin * 2, (cuuint64_t)cin * 2};
        const cuuint32_t box[4] = {16, (cuuint32_t)BN, 3, 9};
        const cuuint32_t estr[4] = {1, 1, 1, 1};
        if (encode(&wmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(w), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return fail("conv: cuTensorMapEncodeTiled rejected the weight layout");
    }
    const int tx = (g.w + S::TX - 1) / S::TX, ty = (g.h + S::TY - 1) / S::TY;
    const long long planes = (long long)(cout / BN) * g.nvol * tx * ty * g.d;
    if (planes >= (1LL << 31)) return 1;
    const int slices = cin / 16, stage = TAPS ? slices * S::ENTRY : S::STAGE;
    // all slices' weights beside the halo stages (tap-major: always; else beside at least four, or a ring of two)
    int wbufs = slices;
    if (!TAPS && (slices > S::MAX_W || slices * S::WSLICE + 4 * stage > kRollSmem)) wbufs = 2;
    int stages = (kRollSmem - wbufs * S::WSLICE) / stage;
    if (stages > (TAPS ? S::MAX_STAGES : 8)) stages = TAPS ? S::MAX_STAGES : 8;
    // a CTA takes all of an SM's tensor memory: more than half its shared memory keeps a second one away
    int smem = wbufs * S::WSLICE + stages * stage;
    if (smem < 120 * 1024) smem = 120 * 1024;
    auto kern = conv3_roll_kernel<BN, TAPS>;
    static std::atomic<unsigned long long> done{0};
    allow_smem(kern, dev, done);
    const int grid = (int)(planes < sms ? planes : sms);
    const int chunk = TAPS || slices == 1 ? g.d : S::R;
    const bool wide = ((reinterpret_cast<uintptr_t>(y)) & 31u) == 0;
    return launch_chained(kern, (unsigned)grid, 320, smem, st, xmap, wmap, bias, mask, y, g, cin, cout, relu, tx, ty, (int)planes,
                          chunk, stages, wbufs, wide ? 1 : 0);
}

// Estimated cycles of a CTA's run of conv3_roll_kernel<bn>: its MMAs (the larger of 3027 multiply-adds and 80 operand
// bytes a cycle, the rates the kernel measured at N = 192 and below) or its copies (a row a cycle), over the planes
// of its run and two halo planes per piece.  Negative where the tap-major order does not fit in shared memory.
double roll_cost(const Geo& g, int cin, int cout, int bn, bool taps, int sms) {
    const int slices = cin / 16, R = 512 / bn;
    const double planes = (double)(cout / bn) * g.nvol * ((g.w + 7) / 8) * ((g.h + 15) / 16) * g.d;
    const double run = ceil(planes / (planes < sms ? planes : sms));
    const double piece = (taps || slices == 1 || g.d < R) ? g.d : R;
    const double pieces = run > piece ? ceil(run / piece) : 1.0;
    const double halo = run + 2.0 * pieces;
    const int n = (int)(run < 3 ? run : 3) * bn;
    const double rate = 128.0 * 16.0 * n / 3027.0, read = 32.0 * (128 + n) / 80.0;
    const double math = 9.0 * slices * halo * (rate > read ? rate : read);
    if (taps) {
        // the weights come first; two halo planes at least, so that one is copied while the other is read
        if (slices > RollShape<16>::MAX_W || kRollSmem - slices * 27 * bn * 32 < 2 * slices * RollShape<16>::ENTRY) return -1.0;
        return math + 27.0 * bn * slices;
    }
    const double copies = slices * (180.0 * halo + 27.0 * bn * pieces);
    return math > copies ? math : copies;
}

// `taps`: the tap-major order.  Returns 1 where no block width fits it, or the launch does not take it.
int conv3_roll_dispatch(const bf16* x, const bf16* w, const float* bias, const bf16* mask, bf16* y, Geo g, int cin,
                        int cout, int relu, bool taps, cudaStream_t st) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int best = 0;
    double cost = 0.0;
    for (int bn : {16, 32, 48, 64}) {
        if (cout % bn) continue;
        const double c = roll_cost(g, cin, cout, bn, taps, sms);
        if (c >= 0.0 && (!best || c < cost)) {
            best = bn;
            cost = c;
        }
    }
#define ROLL(BN)                                                                                            \
    case BN:                                                                                                \
        return taps ? conv3_roll_launch<BN, true>(x, w, bias, mask, y, g, cin, cout, relu, dev, sms, st)    \
                    : conv3_roll_launch<BN, false>(x, w, bias, mask, y, g, cin, cout, relu, dev, sms, st)
    switch (best) {
        ROLL(64);
        ROLL(48);
        ROLL(32);
        ROLL(16);
        default: return 1;
    }
#undef ROLL
}

// Launch of conv3_stream_kernel.  Returns 1 where two halo planes and two weight buffers don't fit (more than 288 input
// channels).  Every size it takes is the faster on it, from one voxel (82 -> 23 us at 192 to 64).
int conv3_stream_launch(const bf16* x, const bf16* w, const float* bias, const bf16* mask, bf16* y, Geo g, int cin,
                        int cout, int relu, cudaStream_t st) {
    using S = StreamShape;
    const int planes = 2 * (cin / 16) * S::ENTRY;
    int wbufs = (kRollSmem - planes) / S::WCHUNK;
    if (planes > kRollSmem || wbufs < 2) return 1;
    if (wbufs > S::MAX_W) wbufs = S::MAX_W;
    const int tx = (g.w + 7) / 8, ty = (g.h + 15) / 16;
    const long long tiles = (long long)(cout / S::BN) * g.nvol * g.d * ty * tx;
    if (tiles >= (1LL << 30)) return 1;
    auto encode = tensor_map_encoder();
    if (!encode) return fail("conv: cuTensorMapEncodeTiled is not available");
    CUtensorMap xmap, wmap;
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    {
        const cuuint64_t dims[5] = {(cuuint64_t)cin, (cuuint64_t)g.w, (cuuint64_t)g.h, (cuuint64_t)g.d, (cuuint64_t)g.nvol};
        const cuuint64_t strides[4] = {(cuuint64_t)cin * 2, (cuuint64_t)g.w * cin * 2, (cuuint64_t)g.h * g.w * cin * 2,
                                       (cuuint64_t)g.d * g.h * g.w * cin * 2};
        const cuuint32_t box[5] = {16, (cuuint32_t)S::HX, 18, 1, 1};
        if (encode(&xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<bf16*>(x), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return fail("conv: cuTensorMapEncodeTiled rejected the activation layout");
    }
    {
        // weights [cout][27][cin]: a box of 64 channels of a tap, rows of output channels
        const cuuint64_t dims[3] = {(cuuint64_t)cin, 27, (cuuint64_t)cout};
        const cuuint64_t strides[2] = {(cuuint64_t)cin * 2, (cuuint64_t)27 * cin * 2};
        const cuuint32_t box[3] = {64, 1, (cuuint32_t)S::BN};
        if (encode(&wmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<bf16*>(w), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return fail("conv: cuTensorMapEncodeTiled rejected the weight layout");
    }
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int smem = wbufs * S::WCHUNK + planes;
    static std::atomic<unsigned long long> done{0};
    allow_smem(conv3_stream_kernel, dev, done);
    return launch_chained(conv3_stream_kernel, (unsigned)(tiles < sms ? tiles : sms), 224, smem, st, xmap, wmap, bias, mask, y, g, cin,
                          cout, relu, tx, ty, (int)tiles, wbufs, (reinterpret_cast<uintptr_t>(y) & 31u) == 0 ? 1 : 0);
}

// Narrow 3x3x3 layers run on tcgen05 unless MCXG_DN_MMA_SYNC=1 selects the warp-level mma.sync
// halo kernel (kept as the measured baseline of the tensor-core port).
bool use_tcgen05() {
    static int v = -1;
    if (v < 0) {
        const char* e = getenv("MCXG_DN_MMA_SYNC");
        v = (e && e[0] == '1') ? 0 : 1;
    }
    return v == 1;
}

int conv_fwd_dispatch(const bf16* x, const bf16* w, const float* bias, const bf16* mask, bf16* y, Geo g, int cin,
                      int cout, int taps, int relu, cudaStream_t st) {
    if (use_tcgen05() && taps == 27 && cin % 16 == 0) {
        // 16, 32, 48, 80, 96 .. outputs sum slice by slice, the wider layers tap by tap: the orders of the kernels
        // this one stands in for, kept because a whole network's bf16 roundings follow from them
        const bool narrow = cout % 32 != 0 || (cout / 32 <= 3 && cout % 64 != 0);
        int rc = conv3_roll_dispatch(x, w, bias, mask, y, g, cin, cout, relu, !narrow, st);
        if (rc == 1 && !narrow && cout % 64 == 0) rc = conv3_stream_launch(x, w, bias, mask, y, g, cin, cout, relu, st);
        if (rc != 1) return rc;
    }
    // narrow 3x3x3 layers: halo tiles (each input voxel loaded once per tile, not once per tap)
    if (taps == 27 && cin % 16 == 0 && cout % 32 == 0 && cout / 32 <= 3 && cout % 64 != 0)
        return conv3_halo_launch<32>(x, w, bias, mask, y, g, cin, cout, relu, st);
    if (taps == 27 && cin % 16 == 0 && cout % 32 != 0)
        return conv3_halo_launch<16>(x, w, bias, mask, y, g, cin, cout, relu, st);
    if (cout % 128 == 0) return conv_fwd_launch<128, 128, 32, 2, 4, 4>(x, w, bias, mask, y, g, cin, cout, taps, relu, st);
    if (cout % 64 == 0) return conv_fwd_launch<128, 64, 32, 4, 2, 4>(x, w, bias, mask, y, g, cin, cout, taps, relu, st);
    if (cout % 32 == 0) return conv_fwd_launch<128, 32, 64, 4, 1, 3>(x, w, bias, mask, y, g, cin, cout, taps, relu, st);
    return conv_fwd_launch<128, 16, 64, 4, 1, 3>(x, w, bias, mask, y, g, cin, cout, taps, relu, st);
}

// Launch of conv3_wgrad_kernel.  Returns 1 where its tiles do not fit (the caller takes the general kernel).  A CTA an
// SM, shared evenly by the groups: fewer CTAs with longer runs, for fewer additions to dW, were never faster (2 x 64^3
// 16 to 16: 50 runs 23 us, 24 runs 38; 4 x 8^3 64 to 128: 32 runs 17.4, 16 runs 16.1, 8 runs 20).
template <int COUT>
int conv3_wgrad_launch(const bf16* dy, const bf16* x, float* dw, Geo g, int cin, cudaStream_t st) {
    using S = WgradShape<COUT>;
    auto encode = tensor_map_encoder();
    if (!encode) return fail("wgrad: cuTensorMapEncodeTiled is not available");
    const int tx = (g.w + 7) / 8, ty = (g.h + 15) / 16, tz = (g.d + S::PZ - 1) / S::PZ;
    const long long tiles = (long long)g.nvol * tx * ty * tz;
    const int pairs = 9 * (cin / 16), groups = (pairs + S::G - 1) / S::G;
    int nsl = 1;
    for (int p = 0; p < pairs; p += S::G) {
        const int n = ((p + S::G < pairs ? p + S::G : pairs) - 1) / 9 - p / 9 + 1;
        nsl = n > nsl ? n : nsl;
    }
    const int stage = S::YBYTES + nsl * S::XSTRIDE;
    int stages = kRollSmem / stage;
    if (stages > S::MAX_STAGES) stages = S::MAX_STAGES;
    if (stages < 2 || tiles >= (1LL << 31)) return 1;
    CUtensorMap maps[2];
    for (int m = 0; m < 2; ++m) {
        // dY [nvol][d][h][w][cout] in boxes of PZ planes of 16 x 8 voxels, X [..][cin] with one voxel more on every side
        const cuuint64_t c = m ? cin : COUT;
        const cuuint64_t dims[5] = {c, (cuuint64_t)g.w, (cuuint64_t)g.h, (cuuint64_t)g.d, (cuuint64_t)g.nvol};
        const cuuint64_t strides[4] = {c * 2, (cuuint64_t)g.w * c * 2, (cuuint64_t)g.h * g.w * c * 2,
                                       (cuuint64_t)g.d * g.h * g.w * c * 2};
        const cuuint32_t box[5] = {16, m ? 10u : 8u, m ? 18u : 16u, (cuuint32_t)(m ? S::PZ + 2 : S::PZ), 1};
        const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
        if (encode(&maps[m], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<bf16*>(m ? x : dy), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return fail("wgrad: cuTensorMapEncodeTiled rejected the layout");
    }
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int parts = sms / groups;
    if (parts < 1) parts = 1;
    if (parts > tiles) parts = (int)tiles;          // no run without a tile: the kernel adds what its run left
    int smem = stages * stage;
    if (smem < 120 * 1024) smem = 120 * 1024;       // one CTA an SM: each takes all of its tensor memory
    auto kern = conv3_wgrad_kernel<COUT>;
    static std::atomic<unsigned long long> done{0};
    allow_smem(kern, dev, done);
    return launch_chained(kern, (unsigned)(groups * parts), 192, smem, st, maps[0], maps[1], dy, x, dw, g, cin, tx, ty, tz, (int)tiles, parts,
                          stages, (reinterpret_cast<uintptr_t>(dw) & 15u) == 0 ? 1 : 0);
}

template <int BM>
int wgrad_launch(const bf16* dy, const bf16* x, float* dw, Geo g, int cin, int taps, cudaStream_t st) {
    constexpr int STAGES = 4;
    constexpr int smem = STAGES * (32 * BM + 32 * 64) * 2;
    auto kern = conv_wgrad_kernel<BM, STAGES>;
    static bool attr = false;
    if (!attr) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        attr = true;
    }
    const int ntiles = (taps * cin + 63) / 64;
    // about 4 CTAs per SM over the (column tile, voxel slice) grid, slices a multiple of 32 voxels
    long long want = 152 * 4 / ntiles;
    if (want < 1) want = 1;
    long long kslice = (g.m + want - 1) / want;
    kslice = ((kslice + 31) / 32) * 32;
    if (kslice < 256) kslice = 256;
    unsigned nsl = (unsigned)((g.m + kslice - 1) / kslice);
    kern<<<dim3((unsigned)ntiles, nsl), 128, smem, st>>>(dy, x, dw, g, cin, taps, kslice);
    return launched();
}

Geo make_geo(int nvol, int d, int h, int w) {
    Geo g;
    g.nvol = nvol;
    g.d = d;
    g.h = h;
    g.w = w;
    g.m = (long long)nvol * d * h * w;
    return g;
}

bool dims_ok(int nvol, int d, int h, int w) { return nvol > 0 && d > 0 && h > 0 && w > 0; }

}  // namespace

extern "C" {

const char* mcxg_dn_last_error(void) { return g_err; }

int mcxg_dn_check(void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        snprintf(g_err, sizeof(g_err), "denoiser stream: %s", cudaGetErrorString(e));
        return -(int)e;
    }
    unsigned f = 0;
    e = cudaMemcpyFromSymbol(&f, g_dn_fault, sizeof(f));
    if (e != cudaSuccess) {
        snprintf(g_err, sizeof(g_err), "denoiser fault word: %s", cudaGetErrorString(e));
        return -(int)e;
    }
    if (f) {
        const unsigned zero = 0;
        cudaMemcpyToSymbol(g_dn_fault, &zero, sizeof(zero));
        return fail("a tensor-core convolution gave up waiting for its MMAs (bounded wait); its output is invalid");
    }
    return 0;
}

int mcxg_dn_conv_fwd(const void* x, const void* w, const float* bias, const void* mask, void* y, int nvol, int d,
                     int h, int wd, int cin, int cout, int taps, int relu, void* stream) {
    if (!x || !w || !y || !dims_ok(nvol, d, h, wd)) return fail("conv: null tensor or empty volume");
    if (cin % 8 || cout % 16 || cin <= 0 || cout <= 0) return fail("conv: cin must be a multiple of 8, cout of 16");
    if (taps != 1 && taps != 27) return fail("conv: taps must be 1 or 27");
    if (!aligned16(x) || !aligned16(w) || !aligned16(y) || (mask && !aligned16(mask)))
        return fail("conv: tensors must be 16-byte aligned");
    Geo g = make_geo(nvol, d, h, wd);
    if (g.m >= (1LL << 31) || d >= 1024 || h >= 1024 || wd >= 1024) return fail("conv: volume too large");
    return conv_fwd_dispatch(static_cast<const bf16*>(x), static_cast<const bf16*>(w), bias,
                             static_cast<const bf16*>(mask), static_cast<bf16*>(y), g, cin, cout, taps, relu,
                             static_cast<cudaStream_t>(stream));
}

int mcxg_dn_conv_wgrad(const void* dy, const void* x, float* dw, int nvol, int d, int h, int wd, int cin, int cout,
                       int taps, void* stream) {
    if (!dy || !x || !dw || !dims_ok(nvol, d, h, wd)) return fail("wgrad: null tensor or empty volume");
    if (cin % 16 || cin <= 0) return fail("wgrad: input channels must be a multiple of 16");
    if (taps != 1 && taps != 27) return fail("wgrad: taps must be 1 or 27");
    if (!aligned16(dy) || !aligned16(x)) return fail("wgrad: tensors must be 16-byte aligned");
    Geo g = make_geo(nvol, d, h, wd);
    auto st = static_cast<cudaStream_t>(stream);
    auto DY = static_cast<const bf16*>(dy);
    auto X = static_cast<const bf16*>(x);
    // The tensor-memory kernel from 2^19 (voxels x input channels) on.  Either side, the general kernel's time against
    // it, device us: 8192 voxels 16 to 16 5.9 / 7.6, 8192 32 to 32 7.9 / 8.8, 2048 128 to 128 13.9 / 18.3; 13547 48 to 16
    // 11.6 / 9.2, 32768 16 to 16 10.3 / 7.7, 16384 64 to 64 22.8 / 13.8, 8192 128 to 128 33.7 / 22.5.  Below it one
    // CTA's fixed costs (its tensor memory, the walk over its accumulators) are the whole time.
    if (taps == 27 && use_tcgen05() && (long long)nvol * d * h * wd * cin >= (1 << 19)) {
        int rc = 1;
        switch (cout) {
            case 16: rc = conv3_wgrad_launch<16>(DY, X, dw, g, cin, st); break;
            case 32: rc = conv3_wgrad_launch<32>(DY, X, dw, g, cin, st); break;
            case 64: rc = conv3_wgrad_launch<64>(DY, X, dw, g, cin, st); break;
            case 128: rc = conv3_wgrad_launch<128>(DY, X, dw, g, cin, st); break;
            default: break;
        }
        if (rc != 1) return rc;
    }
    switch (cout) {
        case 16: return wgrad_launch<16>(DY, X, dw, g, cin, taps, st);
        case 32: return wgrad_launch<32>(DY, X, dw, g, cin, taps, st);
        case 64: return wgrad_launch<64>(DY, X, dw, g, cin, taps, st);
        case 128: return wgrad_launch<128>(DY, X, dw, g, cin, taps, st);
        default: return fail("wgrad: output channels must be 16, 32, 64 or 128");
    }
}

int mcxg_dn_bias_grad(const void* dy, float* db, long long m, int c, void* stream) {
    if (!dy || !db || m <= 0) return fail("bias grad: null tensor or no voxels");
    if (c <= 0 || 256 % c) return fail("bias grad: channels must divide 256");
    if (c % 8 == 0 && aligned16(dy)) {
        // about eight rows a thread, at most four blocks an SM
        const long long rows = 256 / (c / 8), want = (m + 8 * rows - 1) / (8 * rows);
        return launch_chained(bias_grad8_kernel, (unsigned)(want < 608 ? want : 608), 256, 0, static_cast<cudaStream_t>(stream),
                              static_cast<const bf16*>(dy), db, m, c);
    }
    long long rows = 4096;
    unsigned blocks = (unsigned)((m + rows - 1) / rows);
    bias_grad_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const bf16*>(dy), db, m, c, rows);
    return launched();
}

int mcxg_dn_pool(const void* x, void* y, int nvol, int d, int h, int w, int c, void* stream) {
    if (!x || !y || !dims_ok(nvol, d, h, w) || (d | h | w) & 1 || c % 8) return fail("pool: bad shape");
    long long work = (long long)nvol * (d / 2) * (h / 2) * (w / 2) * (c / 8);
    return launch_chained(pool_kernel, (unsigned)grid_for(work, 256), 256, 0, static_cast<cudaStream_t>(stream),
                          static_cast<const bf16*>(x), static_cast<bf16*>(y), nvol, d, h, w, c);
}

int mcxg_dn_upcat(const void* low, const void* skip, void* cat, int nvol, int d, int h, int w, int c1, int c2,
                  void* stream) {
    if (!low || !skip || !cat || !dims_ok(nvol, d, h, w) || (d | h | w) & 1 || c1 % 8 || c2 % 8)
        return fail("upcat: bad shape");
    long long work = (long long)nvol * d * h * w * ((c1 + c2) / 8);
    if (work > 0 && work < (1LL << 31) - 1024 && c1 >= 0 && c2 >= 0) {
        return launch_chained(upcat4_kernel, (unsigned)((work + 1023) / 1024), 256, 0, static_cast<cudaStream_t>(stream),
                              static_cast<const uint4*>(low), static_cast<const uint4*>(skip), static_cast<uint4*>(cat), (unsigned)work,
                              (unsigned)(c1 / 8), FastDiv((unsigned)((c1 + c2) / 8)), FastDiv((unsigned)w), FastDiv((unsigned)h),
                              FastDiv((unsigned)d));
    }
    upcat_kernel<<<grid_for(work, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const bf16*>(low), static_cast<const bf16*>(skip), static_cast<bf16*>(cat), nvol, d, h, w, c1, c2);
    return launched();
}

int mcxg_dn_upcat_bwd(const void* dcat, const void* low, void* dlow, int nvol, int d, int h, int w, int c1, int c2,
                      void* stream) {
    if (!dcat || !low || !dlow || !dims_ok(nvol, d, h, w) || (d | h | w) & 1 || c1 % 8 || c2 % 8)
        return fail("upcat backward: bad shape");
    long long work = (long long)nvol * (d / 2) * (h / 2) * (w / 2) * (c1 / 8);
    upcat_bwd_kernel<<<grid_for(work, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const bf16*>(dcat), static_cast<const bf16*>(low), static_cast<bf16*>(dlow), nvol, d, h, w, c1, c2);
    return launched();
}

int mcxg_dn_unpool_add(const void* dpool, const void* dcat, const void* enc, void* denc, int nvol, int d, int h, int w,
                       int c1, int c, void* stream) {
    if (!dpool || !enc || !denc || !dims_ok(nvol, d, h, w) || (d | h | w) & 1 || c % 8 || c1 % 8)
        return fail("unpool: bad shape");
    long long work = (long long)nvol * d * h * w * (c / 8);
    unpool_add_kernel<<<grid_for(work, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const bf16*>(dpool), static_cast<const bf16*>(dcat), static_cast<const bf16*>(enc),
        static_cast<bf16*>(denc), nvol, d, h, w, c1, c);
    return launched();
}

int mcxg_dn_head(const void* act, const float* xres, const float* w, const float* b, const float* target,
                 const float* valid, float* out, void* dact, float* dw, float* db, float* loss, long long m, float inv,
                 void* stream) {
    if (!act || !xres || !w || !b || m <= 0) return fail("head: null tensor or no voxels");
    if (target && (!valid || !dact || !dw || !db || !loss)) return fail("head: training needs valid/dact/dw/db/loss");
    if (!target && !out) return fail("head: nothing to write");
    return launch_chained(head_kernel, (unsigned)grid_for(m, 256), 256, 0, static_cast<cudaStream_t>(stream),
                          static_cast<const bf16*>(act), xres, w, b, target, valid, out, static_cast<bf16*>(dact), dw, db, loss, m, inv);
}

int mcxg_dn_pack(const float* flux, const uint8_t* label, const float* props, const float* log_photons, void* x0,
                 float* xres, int nvol, int d, int h, int w, int nprop, void* stream) {
    if (!flux || !label || !props || !log_photons || !x0 || !xres || !dims_ok(nvol, d, h, w) || nprop <= 0)
        return fail("pack: bad arguments");
    Geo g = make_geo(nvol, d, h, w);
    // four voxels of a row with one access where every row starts on one
    const int vec = w % 4 == 0 && aligned16(flux) && aligned16(xres) && (reinterpret_cast<uintptr_t>(label) & 3u) == 0;
    // tiles of 64 or of 32 voxels in x, whichever pads less
    auto run = [&](auto kern, int tx) {
        const int tiles_x = (w + 4 * tx - 1) / (4 * tx), y = 128 / tx, tiles_y = (h + y - 1) / y, tiles_z = (d + 3) / 4;
        const long long tiles = (long long)nvol * tiles_z * tiles_y * tiles_x;
        kern<<<(unsigned)(tiles < 0x7fffffff ? tiles : 0x7fffffff), 512, 0, static_cast<cudaStream_t>(stream)>>>(
            flux, label, props, log_photons, static_cast<bf16*>(x0), xres, g, nprop, tiles_x, tiles_y, tiles_z, tiles,
            (reinterpret_cast<uintptr_t>(x0) & 31u) == 0 ? 1 : 0, vec);
        return launched();
    };
    return (w - 1) % 64 < 32 ? run(pack_kernel<8>, 8) : run(pack_kernel<16>, 16);
}

int mcxg_dn_adamw(float* master, float* grad, float* m1, float* m2, void* w16, void* wt16, long long n, int cout,
                  int taps, int cin, float lr, float b1, float b2, float eps, float wd, int step, void* stream) {
    if (!master || !grad || !m1 || !m2 || n <= 0 || step < 1) return fail("adamw: bad arguments");
    if (wt16 && (taps <= 0 || (long long)cout * taps * cin != n)) return fail("adamw: transposed copy needs the shape");
    float bc1 = 1.f - powf(b1, (float)step), bc2 = 1.f - powf(b2, (float)step);
    adamw_kernel<<<grid_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        master, grad, m1, m2, static_cast<bf16*>(w16), static_cast<bf16*>(wt16), n, cout, taps, cin, lr, b1, b2, eps,
        wd, bc1, bc2);
    return launched();
}

}  // extern "C"
