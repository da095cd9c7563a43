// conv3_wgrad.cuh -- weight gradient of the denoiser's 3x3x3 convolutions on the fifth-generation tensor cores.
// Included by denoise.cu inside its namespace.
//
//   dW[co, (dz, dydx), ci] += sum over voxels v of dY[v, co] * X[v + off, ci]
//
// The reduction runs over voxels, so both operands are read "MN-major": a K step is 16 voxels (two y rows of 8
// consecutive x), each a row of 32 bytes (16 channels) as the TMA copy left it, 32-byte swizzle.  M = 128 is PZ z planes x
// Cout of dY (PZ = 128 / Cout), N = (PZ + 2) z planes x 16 channels of X: every pair of planes is formed at once, and the
// pairs whose distance is a tap's dz, 3 PZ of PZ (PZ + 2), are the gradient: 30% of the products at 16 outputs, 50%
// at 32, 75% at 64, all at 128.  The rest is the price of operands wide enough for the tensor cores where a layer
// has 16 channels; mma.sync formed only the useful products and gathered every tap's operands with ldmatrix, at 13%
// of its own peak.  The nine (dy, dx) taps are the same X planes entered at another row.
//
// An accumulator per (slice of 16 input channels, dydx tap), N columns each: tensor memory holds G = 512 / N of them, a
// group.  A CTA takes one group over a run of tiles (16 y x 8 x x PZ z), two or more tiles in flight, and at the end adds
// the diagonals of its accumulators over the planes, through shared memory over its warps, to dW with vector
// reductions.  A sum in tensor memory is as long as the run, eight K steps a tile: 88 at 2 x 64^3 16 to 16, 4096 at 4 x
// 128^3 48 to 16, about a fifth of the general kernel's chains (there, on operands with a mean, it is off by 3.0e-5 of the sum of
// absolute values, the general kernel by 1.5e-4).
//
// Roles: warp 4 issues the copies, warp 5 the MMAs (converged, one elected lane), warps 0-3 the epilogue.  Every wait is
// bounded and reports through g_dn_fault.
//
// Measured (GB300, device us, the mma.sync kernel before against this one): 2 x 64^3 16 to 16 99 / 23, 4 x 64^3 48 to 16
// 592 / 114 (380 TFLOP/s useful, of 1270 formed), 4 x 32^3 32 to 32 53 / 19, 4 x 32^3 96 to 32 153 / 41, 4 x 16^3
// 64 to 64 23 / 14, 32^3 64 to 64 38 / 17, 4 x 16^3 128 to 128 59 / 29.  Bound by the tensor cores' reads of operands
// (an MMA reads 128 x 32 bytes of dY and N x 32 of X for its N columns); at few tiles by the additions to dW.

template <int COUT>
struct WgradShape {
    static constexpr int PZ = 128 / COUT;                 // z planes of dY in M = 128
    static constexpr int N = (PZ + 2) * 16;
    static constexpr int G = 512 / N < 10 ? 512 / N : 10; // accumulators; at most ten, so that a group spans two slices
    static constexpr int YBYTES = 128 * 256;              // dY of a tile: 128 voxels a plane x PZ planes x COUT channels
    static constexpr int XPLANE = 18 * 10 * 32;
    static constexpr int XBYTES = (PZ + 2) * XPLANE;      // a slice of the tile's X planes with their halo
    static constexpr int XSTRIDE = (XBYTES + 1023) / 1024 * 1024;
    static constexpr int MAX_STAGES = 4;
};

// Descriptor of an MN-major operand in the 32-byte swizzle: 16-channel blocks `lbo` bytes apart, groups of 8 voxels `sbo`.
__device__ __forceinline__ uint64_t umma_desc_mn32(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46) | (6ull << 61);
}

// A CTA's group over its run on mma.sync, without the products of voxels outside the volume: for a run whose sums hold an
// infinity or a NaN (below).  The same tiles, copied to shared memory by all threads; a row of X that a voxel of dY outside
// the volume would meet is read as zeros.  A warp holds 16 output channels x three pairs x three dz; where there
// are fewer such units than warps, they share a unit's K steps.  Bound by the copies, which nothing overlaps.  Rare, but a
// training step that meets one infinity should not stall (GB300, us a call: finite, one infinity, X all NaN, and the
// general kernel on any of them): 2 x 65^3 16 to 16 41, 203, 219, 113; 4 x 65^3 48 to 16 181, 950, 1234, 636; 4 x 33^3
// 96 to 32 86, 735, 804, 176; 33^3 64 to 64 33, 189, 227, 49; 4 x 17^3 128 to 128 67, 818, 847, 76.  (A voxel at a time on the
// CUDA cores took 7.7 to 38 ms for one infinity and 14 to 110 for X all NaN.)
template <int COUT>
__device__ __noinline__ void wgrad_within(unsigned char* smem, const bf16* dy, const bf16* x, float* dw, const Geo& g, int cin, int tiles_x,
                                          int tiles_y, int tiles_z, int t_lo, int t_hi, int pair0, int pairs) {
    using S = WgradShape<COUT>;
    constexpr int PZ = S::PZ, WARPS = 6;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int slice0 = pair0 / 9, nsl = (pair0 + pairs - 1) / 9 - slice0 + 1;
    const int xchunks = nsl * (PZ + 2) * 180 * 2;
    uint4* const sy = reinterpret_cast<uint4*>(smem);               // [Cout / 16][PZ][16][8] rows of 32 bytes
    uint4* const sx = sy + S::YBYTES / 16;                          // [nsl][PZ + 2][18][10] rows
    uint4* const zeros = sx + xchunks;                              // a row
    const int trios = (pairs + 2) / 3, units = COUT / 16 * trios, share = units < WARPS ? WARPS / units : 1;
    for (int base = 0; base < units * share; base += WARPS) {
        const int unit = (base + warp) / share, part = (base + warp) % share;
        const bool on = unit < units;
        const int mb = unit / trios, p0 = unit % trios * 3;
        // the blocks of dY that this pass's units hold: the others need not be copied
        const int y_lo = base / share / trios * PZ * 256, y_hi = (min(units - 1, (base + WARPS - 1) / share) / trios + 1) * PZ * 256;
        float acc[3][3][2][4] = {};
        for (int t = t_lo; t < t_hi; ++t) {
            int r = t;
            const int x0 = (r % tiles_x) * 8;
            r /= tiles_x;
            const int y0 = (r % tiles_y) * 16;
            r /= tiles_y;
            const int z0 = (r % tiles_z) * PZ, n = r / tiles_z;
            const auto voxel = [&](int z, int y, int xx) { return (((long long)n * g.d + z) * g.h + y) * g.w + xx; };
            const auto within = [&](int z, int y, int xx) {
                return (unsigned)z < (unsigned)g.d && (unsigned)y < (unsigned)g.h && (unsigned)xx < (unsigned)g.w;
            };
            __syncthreads();        // the tile before has been read
            for (int i = y_lo + tid; i < y_hi; i += 32 * WARPS) {
                const int xx = x0 + (i >> 1) % 8, yy = y0 + (i >> 4) % 16, zz = z0 + (i >> 8) % PZ, c = (i >> 8) / PZ * 16 + (i & 1) * 8;
                const bool in = within(zz, yy, xx);
                cp_async16(smem_addr(sy + i), in ? dy + voxel(zz, yy, xx) * COUT + c : dy, in);
            }
            for (int i = tid; i < xchunks; i += 32 * WARPS) {
                const int v = i >> 1, s = v / (180 * (PZ + 2)), c = (slice0 + s) * 16 + (i & 1) * 8;
                const int xx = x0 - 1 + v % 10, yy = y0 - 1 + v / 10 % 18, zz = z0 - 1 + v / 180 % (PZ + 2);
                const bool in = within(zz, yy, xx);
                cp_async16(smem_addr(sx + i), in ? x + voxel(zz, yy, xx) * cin + c : x, in);
            }
            if (tid < 2) zeros[tid] = make_uint4(0u, 0u, 0u, 0u);
            cp_commit();
            cp_wait<0>();
            __syncthreads();
            for (int k = part; on && k < PZ * 8; k += share) {      // a K step: two y rows of 8 voxels
                const int p = k >> 3, y = (k & 7) * 2, m = lane >> 3, xx = lane & 7;
                if (z0 + p >= g.d) break;
                uint32_t a[4], b[4];
                ldsm_x4_t(smem_addr(sy + (((mb * PZ + p) * 16 + y + (m >> 1)) * 8 + xx) * 2 + (m & 1)), a);
                const bool in = within(z0 + p, y0 + y + (m & 1), x0 + xx);
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const int pair = pair0 + p0 + i, tap = pair % 9;
                    if (p0 + i >= pairs) break;
#pragma unroll
                    for (int dz = 0; dz < 3; ++dz) {
                        const int row = (((pair / 9 - slice0) * (PZ + 2) + p + dz) * 18 + y + (m & 1) + tap / 3) * 10 + xx + tap % 3;
                        ldsm_x4_t(smem_addr((in ? sx + row * 2 : zeros) + (m >> 1)), b);
                        mma_bf16(acc[i][dz][0], a, b[0], b[1]);
                        mma_bf16(acc[i][dz][1], a, b[2], b[3]);
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int pair = pair0 + p0 + i;
            if (!on || p0 + i >= pairs) break;
#pragma unroll
            for (int dz = 0; dz < 3; ++dz)
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int co = mb * 16 + (lane >> 2) + (e >> 1 & 1) * 8, ci = pair / 9 * 16 + (e >> 2) * 8 + (lane & 3) * 2 + (e & 1);
                    atomicAdd(dw + ((long long)co * 27 + dz * 9 + pair % 9) * cin + ci, acc[i][dz][e >> 2][e & 3]);
                }
        }
    }
}

template <int COUT>
__global__ void __launch_bounds__(192, 1) conv3_wgrad_kernel(const __grid_constant__ CUtensorMap ymap,
                                                             const __grid_constant__ CUtensorMap xmap, const bf16* dy,
                                                             const bf16* x, float* dw, Geo g,
                                                             int cin, int tiles_x, int tiles_y, int tiles_z, int tiles, int parts,
                                                             int stages, int vec4) {
    using S = WgradShape<COUT>;
    constexpr int PZ = S::PZ, N = S::N;
    extern __shared__ __align__(1024) unsigned char dyn_smem[];
    __shared__ __align__(8) uint64_t s_bar[2 * S::MAX_STAGES + 1];
    __shared__ uint32_t s_tmem;

    chain_next();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int group = (int)blockIdx.x / parts, part = (int)blockIdx.x % parts;
    const int pair0 = group * S::G, pairs = min(S::G, 9 * (cin / 16) - pair0);    // pair = slice * 9 + dydx
    const int slice0 = pair0 / 9, nsl = (pair0 + pairs - 1) / 9 - slice0 + 1;
    const int t_lo = (int)((long long)tiles * part / parts), t_hi = (int)((long long)tiles * (part + 1) / parts);
    const uint32_t sh = smem_addr(dyn_smem), stage_bytes = S::YBYTES + nsl * S::XSTRIDE;
    const uint32_t full0 = smem_addr(s_bar), empty0 = full0 + 8 * S::MAX_STAGES, done = empty0 + 8 * S::MAX_STAGES;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(&s_tmem)), "n"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    if (tid == 0) {
        for (int i = 0; i < 2 * S::MAX_STAGES + 1; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(full0 + 8 * i));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = __reduce_max_sync(0xffffffffu, s_tmem);

    bool fault = false;
    chain_wait();
    if (warp == 4) {
        const uint32_t lead = elect_lead();
        RollRing st(stages);
        bool used = false;
        for (int t = t_lo; t < t_hi; ++t) {
            if (used && !warp_wait(empty0 + 8 * st.i, st.phase ^ 1u)) {
                fault = true;
                break;
            }
            int r = t;
            const int x0 = (r % tiles_x) * 8;
            r /= tiles_x;
            const int y0 = (r % tiles_y) * 16;
            r /= tiles_y;
            const int z0 = (r % tiles_z) * PZ, n = r / tiles_z;
            const uint32_t bar = full0 + 8 * st.i, dst = sh + st.i * stage_bytes;
            expect_tx(lead, bar, S::YBYTES + nsl * S::XBYTES);
#pragma unroll
            for (int c = 0; c < COUT / 16; ++c) tma_5d(lead, dst + c * PZ * 4096, &ymap, c * 16, x0, y0, z0, n, bar);
            for (int s = 0; s < nsl; ++s)
                tma_5d(lead, dst + S::YBYTES + s * S::XSTRIDE, &xmap, (slice0 + s) * 16, x0 - 1, y0 - 1, z0 - 1, n, bar);
            st.step();
            used |= st.i == 0;
        }
        if (fault) {        // given up: the copies in flight land before the CTA ends
            for (int j = 0; j < stages; ++j, st.step())
                if (used || j >= stages - st.i) mbar_wait(full0 + 8 * st.i, st.phase ^ 1u);
        }
    } else if (warp == 5) {
        const uint32_t lead = elect_lead();
        // FP32 accumulators, BF16 operands, both MN-major
        const uint32_t idesc = umma_idesc_bf16(N) | (1u << 15) | (1u << 16);
        const int first = pair0 % 9 / 3 * 20 + pair0 % 3 * 2;       // row of the group's first tap, in 16-byte units
        RollRing st(stages);
        for (int t = t_lo; t < t_hi; ++t) {
            if (!warp_wait(full0 + 8 * st.i, st.phase)) {
                fault = true;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const uint32_t base = sh + st.i * stage_bytes;
            const uint64_t a0 = umma_desc_mn32(base, 4096, 256), b0 = umma_desc_mn32(base + S::YBYTES, S::XPLANE, 320);
            for (int k = 0; k < 8; ++k) {                   // two y rows a step
                const uint64_t ad = a0 + (uint64_t)(k * 512 / 16);
                const uint32_t accum = (t > t_lo || k > 0) ? 1u : 0u;
                uint64_t bd = b0 + (uint64_t)(k * 2 * 20 + first);
                int dx = pair0 % 3, dy3 = pair0 % 9 / 3;
                for (int p = 0; p < pairs; ++p) {
                    umma_f16(lead, tmem + (uint32_t)(p * N), ad, bd, idesc, accum);
                    bd += 2;                                // the next tap: a voxel on, a y row, or the next slice
                    if (++dx == 3) {
                        dx = 0;
                        bd += 20 - 6;
                        if (++dy3 == 3) {
                            dy3 = 0;
                            bd += S::XSTRIDE / 16 - 60;
                        }
                    }
                }
            }
            umma_commit(lead, empty0 + 8 * st.i);
            st.step();
        }
        umma_commit(lead, done);
    }
    // the stages are free for the sums once every MMA has read them
    const bool reached = warp_wait(done, 0u), ok = __syncthreads_and(reached) != 0;
    fault |= !reached;
    constexpr int CB = PZ > 1 ? 4 : 3;                      // blocks of 16 columns a warp reads of an accumulator
    const int p_low = PZ > 1 ? (2 * warp) % PZ : 0;
    bool plain = true;
    if (ok && (g.w % 8 | g.h % 16 | g.d % PZ) != 0) {
        // A tile that ends outside the volume pairs zeros of dY there with voxels of X inside it, which adds nothing
        // but where X holds an infinity or a NaN.  A run with such a sum is added up over the volume's own pairs (the look
        // at the sums costs no time that shows).
        bool odd = false;
        if (warp < 4) {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            for (int p = 0; p < pairs; ++p) {
#pragma unroll
                for (int c = 0; c < CB; ++c) {
                    uint32_t v[16];
                    tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(p * N + (p_low + c) * 16), v);
#pragma unroll
                    for (int i = 0; i < 16; ++i) odd |= (v[i] & 0x7F800000u) == 0x7F800000u;
                }
            }
        }
        plain = __syncthreads_or(odd) == 0;
        if (!plain) wgrad_within<COUT>(dyn_smem, dy, x, dw, g, cin, tiles_x, tiles_y, tiles_z, t_lo, t_hi, pair0, pairs);
    }
    if (warp < 4 && ok && plain) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        // lane r holds row r: channel co of plane p, which pairs with the X planes p .. p + 2 (columns 16 p ..)
        const int r = warp * 32 + lane;
        const bool high = PZ > 1 && lane >= 16;             // the warp's upper half holds the next plane
        const int co = (r >> 4) / PZ * 16 + (r & 15);
        float* const sums = reinterpret_cast<float*>(dyn_smem);         // [4 warps][16][48] where warps share channels
        constexpr int SHARE = PZ >= 8 ? 4 : PZ >= 4 ? 2 : 1;            // warps that hold the same channels
        for (int p = 0; p < pairs; ++p) {
            uint32_t v[CB * 16];
#pragma unroll
            for (int c = 0; c < CB; ++c)
                tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(p * N + (p_low + c) * 16),
                          *reinterpret_cast<uint32_t(*)[16]>(&v[c * 16]));
            float f[48];
#pragma unroll
            for (int i = 0; i < 48; ++i) f[i] = __uint_as_float(PZ > 1 ? (high ? v[(i + 16) % (CB * 16)] : v[i]) : v[i]);
            if (PZ > 1) {
#pragma unroll
                for (int i = 0; i < 48; ++i) f[i] += __shfl_xor_sync(0xffffffffu, f[i], 16);
            }
            if (SHARE > 1) {
                // sums[i][warp][channel]: conflict-free, and the four warps' parts side by side
                asm volatile("bar.sync 1, 128;\n" ::: "memory");
                if (lane < 16) {
#pragma unroll
                    for (int i = 0; i < 48; ++i) sums[(i * 4 + warp) * 16 + lane] = f[i];
                }
                asm volatile("bar.sync 1, 128;\n" ::: "memory");
                if (warp % SHARE == 0 && lane < 16) {
#pragma unroll
                    for (int i = 0; i < 48; ++i)
#pragma unroll
                        for (int q = 1; q < SHARE; ++q) f[i] += sums[(i * 4 + warp + q) * 16 + lane];
                }
            }
            const bool mine = PZ == 1 || ((warp % SHARE) == 0 && lane < 16);
            if (mine) {
                const int pair = pair0 + p, sl = pair / 9, tap = pair % 9;
#pragma unroll
                for (int dz = 0; dz < 3; ++dz) {
                    float* o = dw + ((long long)co * 27 + dz * 9 + tap) * cin + sl * 16;
                    if (vec4) {
#pragma unroll
                        for (int i = 0; i < 16; i += 4)
                            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(o + i), "f"(f[dz * 16 + i]),
                                         "f"(f[dz * 16 + i + 1]), "f"(f[dz * 16 + i + 2]), "f"(f[dz * 16 + i + 3])
                                         : "memory");
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i) atomicAdd(o + i, f[dz * 16 + i]);
                    }
                }
            }
        }
    }
    if (fault && lane == 0) atomicOr(&g_dn_fault, 1u);
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "n"(512));
}
