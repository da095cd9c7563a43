// conv3_stream.cuh -- 3x3x3 convolution of the denoiser's widest inputs (more channels than a tap-major conv3_roll_kernel
// keeps weights for) on the fifth-generation tensor cores, weights streamed.  Included by denoise.cu inside its namespace.
//
// A tile is one plane of 16 y x 8 x voxels (M = 128) and 64 output channels.  Sums run tap by tap, within a tap by
// ascending channels: the order of the kernel this one stands in for, so the bits are the same.  Per tap plane dz the halo
// of 18 x 10 voxels, all channels, is copied once and serves the nine (dy, dx) taps as an operand entered at another row
// (32-byte rows and swizzle, as in conv3_roll.cuh); two such buffers, so one is copied while the other is read.  The
// weights of a tap and 64 channels (64 rows of 128 bytes, 128-byte swizzle) pass through a ring of 8 KB buffers: they
// don't fit beside the halo (663 KB at 192 to 64), every CTA reads them from L2 once per tile.  Two accumulators, so a
// tile's epilogue overlaps the next tile's MMAs.
//
// Roles: warps 0-3 epilogue, warp 4 copies planes, warp 5 weights, warp 6 issues the MMAs.  Every wait is bounded and
// reports through g_dn_fault.
//
// Measured (GB300, us, the mma.sync kernel before -> this one): 192 -> 64 at one voxel to 4 x 16^3 82 -> 23, at 32^3
// 118 -> 42, 4 x 32^3 383 -> 133; 256 -> 128 at 16^3 136 -> 29; 160 -> 192 at 32^3 272 -> 108.  A tile takes 18 us, 105
// cycles an MMA against 77 for its operand reads (128 + 64 rows of 32 bytes, 80 bytes a cycle); 256 tiles at 32^3 are 1.7
// waves.

struct StreamShape {
    static constexpr int BN = 64, HX = 10, ZPLANE = 18 * HX * 32, ENTRY = 5888;
    static constexpr int WCHUNK = BN * 128, MAX_W = 16;
};

// Descriptor of a K-major operand of 128-byte rows in the 128-byte swizzle, 8-row groups 1 KB apart.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

// A CTA's tiles, grid apart: the same sequence for every role.
struct StreamTile {
    int t, tiles, tx, ty, d, nvol;
    int n0, n, z, y0, x0;
    __device__ __forceinline__ StreamTile(int tiles_, int tx_, int ty_, const Geo& g)
        : t((int)blockIdx.x - (int)gridDim.x), tiles(tiles_), tx(tx_), ty(ty_), d(g.d), nvol(g.nvol) {
        n0 = n = z = y0 = x0 = 0;
    }
    __device__ __forceinline__ bool next() {
        if (t >= tiles - (int)gridDim.x) return false;
        t += gridDim.x;
        int r = t;
        x0 = (r % tx) * 8;
        r /= tx;
        y0 = (r % ty) * 16;
        r /= ty;
        z = r % d;
        r /= d;
        n = r % nvol;
        n0 = r / nvol * StreamShape::BN;
        return true;
    }
};

__global__ void __launch_bounds__(224, 1) conv3_stream_kernel(const __grid_constant__ CUtensorMap xmap,
                                                              const __grid_constant__ CUtensorMap wmap,
                                                              const float* bias, const bf16* mask, bf16* y, Geo g, int cin, int cout, int relu, int tiles_x,
                                                              int tiles_y, int tiles, int wbufs, int wide) {
    using S = StreamShape;
    constexpr int BN = S::BN;
    extern __shared__ __align__(1024) unsigned char dyn_smem[];
    __shared__ __align__(8) uint64_t s_bar[2 * S::MAX_W + 8];
    __shared__ uint32_t s_tmem;

    chain_next();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int slices = cin / 16, chunks = (cin + 63) / 64;
    const uint32_t sw = smem_addr(dyn_smem), sh = sw + wbufs * S::WCHUNK, plane = slices * S::ENTRY;
    const uint32_t wfull0 = smem_addr(s_bar), wempty0 = wfull0 + 8 * S::MAX_W, pfull0 = wempty0 + 8 * S::MAX_W, pempty0 = pfull0 + 16,
                   afull0 = pempty0 + 16, aempty0 = afull0 + 16;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(&s_tmem)), "n"(2 * BN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    if (tid == 0) {
        // arrivals: one (a copy's expect, an MMA commit), but four warps free an accumulator
        for (int i = 0; i < 2 * S::MAX_W + 6; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(wfull0 + 8 * i));
        for (int i = 0; i < 2; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;\n" ::"r"(aempty0 + 8 * i));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = __reduce_max_sync(0xffffffffu, s_tmem);

    bool fault = false;
    StreamTile tile(tiles, tiles_x, tiles_y, g);
    chain_wait();
    if (warp == 4) {
        const uint32_t lead = elect_lead();
        RollRing st(2);
        bool used = false;
        while (!fault && tile.next()) {
            for (int dz = 0; dz < 3; ++dz) {
                if (used && !warp_wait(pempty0 + 8 * st.i, st.phase ^ 1u)) {
                    fault = true;
                    break;
                }
                const uint32_t bar = pfull0 + 8 * st.i;
                expect_tx(lead, bar, slices * S::ZPLANE);
                for (int sl = 0; sl < slices; ++sl)
                    tma_5d(lead, sh + st.i * plane + sl * S::ENTRY, &xmap, sl * 16, tile.x0 - 1, tile.y0 - 1, tile.z - 1 + dz, tile.n, bar);
                st.step();
                used |= st.i == 0;
            }
        }
        if (fault) {        // given up: the copies in flight land before the CTA ends
            for (int j = 0; j < 2; ++j, st.step())
                if (used || j >= 2 - st.i) mbar_wait(pfull0 + 8 * st.i, st.phase ^ 1u);
        }
    } else if (warp == 5) {
        const uint32_t lead = elect_lead();
        RollRing st(wbufs);
        bool used = false;
        while (!fault && tile.next()) {
            for (int t = 0; t < 27 && !fault; ++t)
                for (int c = 0; c < chunks; ++c) {
                    if (used && !warp_wait(wempty0 + 8 * st.i, st.phase ^ 1u)) {
                        fault = true;
                        break;
                    }
                    const uint32_t bar = wfull0 + 8 * st.i;
                    expect_tx(lead, bar, S::WCHUNK);
                    tma_3d(lead, sw + st.i * S::WCHUNK, &wmap, c * 64, t, tile.n0, bar);
                    st.step();
                    used |= st.i == 0;
                }
        }
        if (fault) {
            for (int j = 0; j < wbufs; ++j, st.step())
                if (used || j >= wbufs - st.i) mbar_wait(wfull0 + 8 * st.i, st.phase ^ 1u);
        }
    } else if (warp == 6) {
        const uint32_t lead = elect_lead();
        constexpr uint32_t idesc = umma_idesc_bf16(BN);
        RollRing st(2), wr(wbufs), acc(2);
        bool used = false;
        while (!fault && tile.next()) {
            if (used && !warp_wait(aempty0 + 8 * acc.i, acc.phase ^ 1u)) {
                fault = true;
                break;
            }
            const uint32_t d = tmem + (uint32_t)(acc.i * BN);
            uint32_t accum = 0u;
            for (int dz = 0; dz < 3 && !fault; ++dz) {
                if (!warp_wait(pfull0 + 8 * st.i, st.phase)) {
                    fault = true;
                    break;
                }
                const uint64_t a0 = umma_desc_sw32(sh + st.i * plane, S::HX * 32);
                for (int t = 0; t < 9 && !fault; ++t) {
                    uint64_t ad = a0 + (uint64_t)(2 * ((t / 3) * S::HX + t % 3));
                    for (int c = 0; c < chunks; ++c) {
                        if (!warp_wait(wfull0 + 8 * wr.i, wr.phase)) {
                            fault = true;
                            break;
                        }
                        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                        uint64_t bd = umma_desc_sw128(sw + wr.i * S::WCHUNK);
                        const int ns = min(4, slices - 4 * c);
                        for (int k = 0; k < ns; ++k, ad += S::ENTRY / 16, bd += 2, accum = 1u) umma_f16(lead, d, ad, bd, idesc, accum);
                        umma_commit(lead, wempty0 + 8 * wr.i);
                        wr.step();
                    }
                }
                umma_commit(lead, pempty0 + 8 * st.i);
                st.step();
            }
            umma_commit(lead, afull0 + 8 * acc.i);
            acc.step();
            used |= acc.i == 0;
        }
    } else {
        const int r = warp * 32 + lane;                     // accumulator row = TMEM lane = voxel of the plane
        const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
        RollRing acc(2);
        while (tile.next()) {
            if (!warp_wait(afull0 + 8 * acc.i, acc.phase)) {
                fault = true;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            uint32_t v[BN];
#pragma unroll
            for (int c0 = 0; c0 < BN; c0 += 16) tmem_ld16(trow + acc.i * BN + c0, *reinterpret_cast<uint32_t(*)[16]>(&v[c0]));
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(aempty0 + 8 * acc.i);
            acc.step();
            const int yy = tile.y0 + (r >> 3), xx = tile.x0 + (r & 7);
            if (yy < g.h && xx < g.w) {
                const long long at = ((((long long)tile.n * g.d + tile.z) * g.h + yy) * g.w + xx) * cout + tile.n0;
                float bs[BN];
#pragma unroll
                for (int c = 0; c < BN; ++c) bs[c] = bias ? bias[tile.n0 + c] : 0.f;
                uint32_t mk[BN / 2];
                if (mask) {
#pragma unroll
                    for (int c0 = 0; c0 < BN; c0 += 16) roll_mask16(mask + at + c0, mk + c0 / 2);
                }
#pragma unroll
                for (int c0 = 0; c0 < BN; c0 += 16)
                    roll_store16(v + c0, bs + c0, mask ? mk + c0 / 2 : nullptr, y + at + c0, relu, wide != 0);
            }
        }
    }
    if (fault && lane == 0) atomicOr(&g_dn_fault, 1u);
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "n"(2 * BN));
}
