// conv3_roll.cuh -- 3x3x3 convolution (forward and data gradient) of the denoiser on the fifth-generation tensor
// cores, with output planes rolling through tensor memory.  Included by denoise.cu inside its namespace.
//
// A work unit is a column: 16 y rows x 8 x voxels (one M = 128 MMA per plane), running along z, for a block of BN
// output channels.  The halo plane of 18 x 10 voxels around the column at depth z, one 16-channel slice of the
// input, contributes to the output planes z - 1, z, z + 1 through the taps dz = 2, 1, 0.  Those three accumulators lie
// side by side in tensor memory, so each of the nine (dy, dx) taps is ONE MMA of N = 3 BN columns: the A operand (the
// halo seen through a descriptor that starts at the tap's row) is read from shared memory once for three taps.  With
// an MMA per tap (N = BN) the narrow layers were bound by those reads and by the issue of their MMAs.
// The accumulators of the planes form a ring of R = 512 / BN slots (descending columns as z ascends, which puts the
// weights of a tap in dz order); slots are handed over in pairs, drained as soon as their third contribution is in,
// so epilogues overlap the MMAs of the planes behind, and left at zero, so every MMA adds.
//
// Two orders of summation, each the order of the kernel it stands in for, because the bf16 roundings of a whole
// network follow from the order (mma.sync and tcgen05 give the same bits for the same order of K = 16 steps):
//   slice by slice (16, 32, 48, 80, 96 .. outputs): a pass over the run's planes per 16-channel slice;
//   tap by tap (TAPS; the wider layers): per halo plane the nine taps, per tap the slices.
//
// The column sequence (channel block, volume, y, x) x z is cut into one contiguous run of planes per SM, so the
// load is even whatever the sizes, and a run pays two halo planes more per column it touches.  Slice by slice a run in
// several slices keeps all its planes' accumulators at once and is cut into pieces of at most R planes.
//
// Roles: warps 0-7 drain accumulators (two warpgroups, pair by pair in turn), warp 8 issues the TMA copies, warp 9
// the MMAs.  Halo planes and weights arrive as rows of 32 bytes (16 channels of a voxel, or of a tap's output channel) in
// the 32-byte swizzle, out-of-volume rows zero: the K-major operand layout, which a descriptor may enter at any row
// because the swizzle goes by the address.  (8-channel boxes of 16-byte rows, without a swizzle, cost a copied row and
// half an L2 sector each: the copy engine moves about a row a cycle and bound the wide layers, 35 against 27 us for 64 ->
// 64 at 4 x 32^3.)  The weights of all slices stay in shared memory when they fit beside the halo stages (always, tap by
// tap), else they cycle through a ring of slice buffers.  Every wait is bounded: one that gives up sets g_dn_fault, and
// the CTA still releases its tensor memory and returns.
//
// Measured (GB300, us, the kernel before -> this one): 16 -> 16 at 128^3 77 -> 42; 48 -> 16 206 -> 117; 16 -> 48 206 -> 60
// (1460 TFLOP/s, 77% of the measured peak); 32 -> 32 at 64^3 33 -> 17; 96 -> 32 82 -> 40; 64 -> 64 at 4 x 32^3 134 -> 34;
// 64 -> 192 at 32^3 115 -> 25; 128 -> 128 at 16^3 72 -> 15 (back to back, launches overlapping).  What bounds it: operand reads, about 80 bytes a cycle
// (70 cycles per MMA of N = 48), up to N = 144; the math at N = 192; beyond that a fixed 5 us (launch, tensor
// memory, first weights and halo).

template <int BN>
struct RollShape {
    static constexpr int TY = 16, TX = 8, HY = TY + 2, HX = TX + 2;
    static constexpr int ZPLANE = HY * HX * 32;               // a halo plane: rows of 16 channels
    static constexpr int STAGE = 2 * ZPLANE;
    static constexpr int ENTRY = 5888;                        // a slice of one halo plane, padded to 256 (tap-major order)
    static constexpr int N3 = 3 * BN;
    static constexpr int WSLICE = 9 * N3 * 32;                // a slice's weights
    static constexpr int R = 512 / BN, RP = R / 2;            // accumulator slots, and pairs of them
    static constexpr int MAX_STAGES = 12, MAX_W = 12;
};

// Descriptor of a K-major operand of 32-byte rows (16 channels) in the 32-byte swizzle, 8-row groups `sbo` bytes apart.
__device__ __forceinline__ uint64_t umma_desc_sw32(uint32_t saddr, uint32_t sbo) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46) |
           (6ull << 61);
}

// A CTA's run of planes, piece by piece: the same sequence for every role.
struct RollRun {
    int pos, end, d, nvol, ty, tx, chunk, bn;
    int n0, n, y0, x0, z0, nz;          // the current piece
    __device__ __forceinline__ RollRun(int planes, const Geo& g, int ty_, int tx_, int chunk_, int bn_)
        : d(g.d), nvol(g.nvol), ty(ty_), tx(tx_), chunk(chunk_), bn(bn_) {
        pos = (int)((long long)blockIdx.x * planes / gridDim.x);
        end = (int)((long long)(blockIdx.x + 1) * planes / gridDim.x);
        n0 = n = y0 = x0 = z0 = nz = 0;
    }
    __device__ __forceinline__ int block_of(int p) const { return p / d / tx / ty / nvol * bn; }
    __device__ __forceinline__ bool next() {
        pos += nz;
        if (pos >= end) return false;
        int col = pos / d;
        z0 = pos - col * d;
        const int len = min(end - pos, d - z0), pieces = (len + chunk - 1) / chunk;
        nz = (len + pieces - 1) / pieces;
        x0 = (col % tx) * 8;
        col /= tx;
        y0 = (col % ty) * 16;
        col /= ty;
        n = col % nvol;
        n0 = col / nvol * bn;
        return true;
    }
};

// The issuing warps run converged and only their instructions are predicated on one elected lane (`lead`), so that
// descriptors, addresses and counters live in uniform registers.  Issued from inside an `if (lane == 0)` an MMA took
// some 110 cycles of one thread's scalar work, which bound every layer.
__device__ __forceinline__ uint32_t elect_lead() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\tselp.u32 %0, 1, 0, e;\n\t}\n" : "=r"(p));
    return p;
}
__device__ __forceinline__ void umma_f16(uint32_t lead, uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 e, %5, 0;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
        "l"(ad), "l"(bd), "r"(idesc), "r"(accum), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t lead, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %1, 0;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}\n" ::"r"(bar), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void tma_5d(uint32_t lead, uint32_t dst, const CUtensorMap* map, int c, int x, int y, int z, int n,
                                       uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %8, 0;\n\t"
        "@e cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], "
        "[%7];\n\t}\n" ::"r"(dst),
        "l"(map), "r"(c), "r"(x), "r"(y), "r"(z), "r"(n), "r"(bar), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void tma_4d(uint32_t lead, uint32_t dst, const CUtensorMap* map, int a, int b, int c, int d,
                                       uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %7, 0;\n\t"
        "@e cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];\n\t}\n" ::"r"(dst),
        "l"(map), "r"(a), "r"(b), "r"(c), "r"(d), "r"(bar), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void tma_3d(uint32_t lead, uint32_t dst, const CUtensorMap* map, int a, int b, int c, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %6, 0;\n\t"
        "@e cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];\n\t}\n" ::"r"(dst),
        "l"(map), "r"(a), "r"(b), "r"(c), "r"(bar), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void expect_tx(uint32_t lead, uint32_t bar, uint32_t bytes) {
    asm volatile(
        "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %2, 0;\n\t"
        "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}\n" ::"r"(bar), "r"(bytes), "r"(lead)
        : "memory");
}
// A warp's bounded wait, the same answer in every lane; the clock is read only where the phase is still open.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (__all_sync(0xffffffffu, ok != 0u)) return true;
    return __all_sync(0xffffffffu, mbar_wait(bar, parity));
}
__device__ __forceinline__ void tmem_zero16(uint32_t taddr) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};\n" ::"r"(taddr), "r"(0u)
        : "memory");
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
// A ring of buffers walked one by one: index and the parity of the phase its next use completes.
struct RollRing {
    int i = 0, n;
    uint32_t phase = 0;
    __device__ __forceinline__ explicit RollRing(int size) : n(size) {}
    __device__ __forceinline__ void step() {
        if (++i == n) {
            i = 0;
            phase ^= 1u;
        }
    }
};

// 16 channels of the mask.  An ordinary load, and no kernel that is launched chained declares the mask or the bias
// __restrict__: the kernel ahead may write them after this one has started (chain_wait), so they are not read-only for its
// lifetime, as the read-only path needs.
__device__ __forceinline__ void roll_mask16(const bf16* mask, uint32_t* mk) {
    *reinterpret_cast<uint4*>(mk) = *reinterpret_cast<const uint4*>(mask);
    *reinterpret_cast<uint4*>(mk + 4) = *(reinterpret_cast<const uint4*>(mask) + 1);
}

// 16 consecutive bf16 outputs of a voxel: bias, ReLU, the mask's 16 values (or null), and one 32-byte store (two of 16
// where the tensors are aligned to 16 bytes only).
__device__ __forceinline__ void roll_store16(const uint32_t* v, const float* bias, const uint32_t* mk, bf16* y, int relu, bool wide) {
    uint32_t pk[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        float a = __uint_as_float(v[2 * e]) + bias[2 * e], b = __uint_as_float(v[2 * e + 1]) + bias[2 * e + 1];
        if (relu) {
            a = fmaxf(a, 0.f);
            b = fmaxf(b, 0.f);
        }
        __nv_bfloat162 h2 = __floats2bfloat162_rn(a, b);
        pk[e] = *reinterpret_cast<uint32_t*>(&h2);
    }
    if (mk) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            // keep each bf16 where the mask's bf16 is > 0 (sign bit clear and not +0)
            const uint32_t lo = mk[e] & 0xFFFFu, hi = mk[e] >> 16;
            pk[e] &= ((lo & 0x8000u) == 0 && lo != 0 ? 0xFFFFu : 0u) | ((hi & 0x8000u) == 0 && hi != 0 ? 0xFFFF0000u : 0u);
        }
    }
    if (wide) {
        asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"l"(y), "r"(pk[0]), "r"(pk[1]), "r"(pk[2]),
                     "r"(pk[3]), "r"(pk[4]), "r"(pk[5]), "r"(pk[6]), "r"(pk[7])
                     : "memory");
    } else {
        *reinterpret_cast<uint4*>(y) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        *reinterpret_cast<uint4*>(y + 8) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
    }
}

template <int BN, bool TAPS>
__global__ void __launch_bounds__(320, 1) conv3_roll_kernel(const __grid_constant__ CUtensorMap xmap,
                                                            const __grid_constant__ CUtensorMap wmap,
                                                            const float* bias, const bf16* mask, bf16* y, Geo g, int cin, int cout, int relu, int tiles_x,
                                                            int tiles_y, int planes, int chunk, int stages, int wbufs, int wide) {
    using S = RollShape<BN>;
    constexpr int R = S::R, RP = S::RP;
    static_assert(R % 2 == 0 && S::WSLICE % 256 == 0 && S::STAGE % 256 == 0 && S::ENTRY % 256 == 0, "TMA / UMMA alignment");
    extern __shared__ __align__(1024) unsigned char dyn_smem[];
    __shared__ __align__(8) uint64_t s_bar[2 * S::MAX_STAGES + 2 * S::MAX_W + 2 * RP];
    __shared__ uint32_t s_tmem;

    chain_next();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int slices = cin / 16;
    const bool resident = wbufs >= slices;
    const uint32_t sw = smem_addr(dyn_smem), sh = sw + wbufs * S::WSLICE;
    const uint32_t full0 = smem_addr(s_bar), empty0 = full0 + 8 * S::MAX_STAGES, wfull0 = empty0 + 8 * S::MAX_STAGES,
                   wempty0 = wfull0 + 8 * S::MAX_W, pfull0 = wempty0 + 8 * S::MAX_W, pempty0 = pfull0 + 8 * RP;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(&s_tmem)), "n"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    if (tid == 0) {
        // arrivals: one (a copy's expect, an MMA commit), but four warps free a pair of accumulators
        for (int i = 0; i < 2 * S::MAX_STAGES + 2 * S::MAX_W + RP; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(full0 + 8 * i));
        for (int i = 0; i < RP; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;\n" ::"r"(pempty0 + 8 * i));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = __reduce_max_sync(0xffffffffu, s_tmem);
    if (warp < 4) {
        // every accumulator starts at zero and is left at zero by the epilogue, so that every MMA adds
        for (int c = 0; c < 512; c += 16) tmem_zero16(tmem + ((uint32_t)(warp * 32) << 16) + c);
        tmem_store_wait();
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");

    bool fault = false;
    RollRun run(planes, g, tiles_y, tiles_x, chunk, BN);
    chain_wait();
    if (TAPS && warp == 8) {
        // ---- TMA copies, tap-major: every slice's weights, then halo planes slice by slice ------------
        const uint32_t lead = elect_lead();
        RollRing st(stages), slot(RP);
        int held = -1;
        bool st_used = false, slot_used = false, loaded = false;
        uint32_t wphase = 0;
        while (!fault && run.next()) {
            if (held != run.n0) {
                // the weights of a channel block replace the block's before it
                if (loaded && !warp_wait(wempty0, wphase)) {
                    fault = true;
                    break;
                }
                if (loaded) wphase ^= 1u;
                held = run.n0;
                loaded = true;
                for (int sl = 0; sl < slices; ++sl) {
                    expect_tx(lead, wfull0 + 8 * sl, S::WSLICE);
                    tma_4d(lead, sw + sl * S::WSLICE, &wmap, sl * 16, run.n0, 0, 0, wfull0 + 8 * sl);
                }
            }
            for (int i = 0; i < run.nz + 2 && !fault; ++i) {
                if ((i & 1) == 0 && i < run.nz) {
                    if (slot_used && !warp_wait(pempty0 + 8 * slot.i, slot.phase ^ 1u)) {
                        fault = true;
                        break;
                    }
                    slot.step();
                    slot_used |= slot.i == 0;
                }
                if (st_used && !warp_wait(empty0 + 8 * st.i, st.phase ^ 1u)) {
                    fault = true;
                    break;
                }
                const uint32_t bar = full0 + 8 * st.i, dst = sh + st.i * slices * S::ENTRY;
                expect_tx(lead, bar, slices * S::ZPLANE);
                for (int sl = 0; sl < slices; ++sl)
                    tma_5d(lead, dst + sl * S::ENTRY, &xmap, sl * 16, run.x0 - 1, run.y0 - 1, run.z0 - 1 + i, run.n, bar);
                st.step();
                st_used |= st.i == 0;
            }
        }
        if (fault) {        // given up: the copies in flight land before the CTA ends (as below)
            for (int j = 0; j < stages; ++j, st.step())
                if (st_used || j >= stages - st.i) mbar_wait(full0 + 8 * st.i, st.phase ^ 1u);
            for (int sl = 0; loaded && sl < slices; ++sl) mbar_wait(wfull0 + 8 * sl, wphase);
        }
    } else if (TAPS && warp == 9) {
        // ---- MMA issue, tap-major: per halo plane the nine taps, per tap the slices ----------------------
        const uint32_t lead = elect_lead();
        RollRing st(stages), slot(RP);
        int held = -1;
        uint32_t wphase = 1;
        while (!fault && run.next()) {
            const bool reload = held != run.n0;
            held = run.n0;
            if (reload) wphase ^= 1u;
            const int after = run.pos + run.nz;
            RollRing done = slot;
            int s0 = 2 * slot.i;                            // the slot of output plane i of halo plane i (even i)
            for (int i = 0; i < run.nz + 2 && !fault; ++i) {
                const int hi = min(i, run.nz - 1), lo = max(i - 2, 0), cnt = hi - lo + 1, dz0 = i - hi;
                int s = s0 + (i & 1) - dz0;
                if (s < 0) s += R;
                const int n1 = min(cnt, s + 1), n2 = cnt - n1;
                const uint32_t d1 = tmem + (uint32_t)((R - 1 - s) * BN);
                const uint32_t id1 = umma_idesc_bf16(n1 * BN), id2 = umma_idesc_bf16(n2 > 0 ? n2 * BN : BN);
                if (!warp_wait(full0 + 8 * st.i, st.phase)) {
                    fault = true;
                    break;
                }
                for (int sl = 0; reload && i == 0 && sl < slices; ++sl) fault |= !warp_wait(wfull0 + 8 * sl, wphase);
                if (fault) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint64_t a0 = umma_desc_sw32(sh + st.i * slices * S::ENTRY, S::HX * 32);
                const uint64_t b0 = umma_desc_sw32(sw, 256) + (uint64_t)(2 * dz0 * BN);
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    uint64_t ad = a0 + (uint64_t)(2 * ((t / 3) * S::HX + t % 3)), bd = b0 + (uint64_t)(2 * t * S::N3);
#pragma unroll 4
                    for (int sl = 0; sl < slices; ++sl, ad += S::ENTRY / 16, bd += S::WSLICE / 16) umma_f16(lead, d1, ad, bd, id1, 1u);
                }
                if (n2 > 0) {
#pragma unroll
                    for (int t = 0; t < 9; ++t) {
                        uint64_t ad = a0 + (uint64_t)(2 * ((t / 3) * S::HX + t % 3)), bd = b0 + (uint64_t)(2 * (t * S::N3 + n1 * BN));
                        for (int sl = 0; sl < slices; ++sl, ad += S::ENTRY / 16, bd += S::WSLICE / 16) umma_f16(lead, tmem, ad, bd, id2, 1u);
                    }
                }
                umma_commit(lead, empty0 + 8 * st.i);
                st.step();
                if (i & 1) s0 = s0 + 2 == R ? 0 : s0 + 2;
                if (i >= 2 && ((i & 1) || i == run.nz + 1)) {       // output plane i - 2 ends its pair
                    umma_commit(lead, pfull0 + 8 * done.i);
                    done.step();
                }
            }
            if (after < run.end && run.block_of(after) != run.n0) umma_commit(lead, wempty0);
            slot = done;
        }
    } else if (warp == 8) {
        // ---- TMA copies --------------------------------------------------------------------------
        const uint32_t lead = elect_lead();
        RollRing st(stages), wr(wbufs), slot(RP);
        int held = -1;                      // channel block whose weights stay (resident)
        bool st_used = false, wr_used = false, slot_used = false;       // the ring has gone round once
        while (!fault && run.next()) {
            const bool reload = !resident || held != run.n0;
            held = run.n0;
            const int opens = (run.nz + 1) / 2, pairs = run.nz / 2 + 1 + (run.nz & 1);     // ceil((nz + 2) / 2)
            for (int sl = 0; sl < slices && !fault; ++sl) {
                if (reload) {
                    if (wr_used && !warp_wait(wempty0 + 8 * wr.i, wr.phase ^ 1u)) {
                        fault = true;
                        break;
                    }
                    const uint32_t bar = wfull0 + 8 * wr.i, dst = sw + wr.i * S::WSLICE;
                    expect_tx(lead, bar, S::WSLICE);
                    tma_4d(lead, dst, &wmap, sl * 16, run.n0, 0, 0, bar);
                    wr.step();
                    wr_used |= wr.i == 0;
                }
                for (int p = 0; p < pairs; ++p) {
                    // a halo pair that opens two output planes waits for their accumulators here, off the MMA
                    // warp's path: its MMAs start when the pair has landed
                    if (sl == 0 && p < opens) {
                        if (slot_used && !warp_wait(pempty0 + 8 * slot.i, slot.phase ^ 1u)) {
                            fault = true;
                            break;
                        }
                        slot.step();
                        slot_used |= slot.i == 0;
                    }
                    if (st_used && !warp_wait(empty0 + 8 * st.i, st.phase ^ 1u)) {
                        fault = true;
                        break;
                    }
                    const uint32_t bar = full0 + 8 * st.i, dst = sh + st.i * S::STAGE;
                    expect_tx(lead, bar, S::STAGE);
                    tma_5d(lead, dst, &xmap, sl * 16, run.x0 - 1, run.y0 - 1, run.z0 - 1 + 2 * p, run.n, bar);
                    st.step();
                    st_used |= st.i == 0;
                }
            }
        }
        if (fault) {
            // given up: the copies in flight land before the CTA ends.  A buffer's last copy completed the phase
            // before the one its next use would
            for (int j = 0; j < stages; ++j, st.step())
                if (st_used || j >= stages - st.i) mbar_wait(full0 + 8 * st.i, st.phase ^ 1u);
            for (int j = 0; j < wbufs; ++j, wr.step())
                if (wr_used || j >= wbufs - wr.i) mbar_wait(wfull0 + 8 * wr.i, wr.phase ^ 1u);
        }
    } else if (warp == 9) {
        // ---- MMA issue ---------------------------------------------------------------------------
        const uint32_t lead = elect_lead();
        RollRing st(stages), wr(wbufs), slot(RP);   // slot: the ring position of the piece's first pair of planes
        int held = -1;
        while (!fault && run.next()) {
            const bool reload = !resident || held != run.n0;
            held = run.n0;
            if (resident && !reload) wr.phase ^= 1u;        // the same loads again, one round of the ring back
            const int after = run.pos + run.nz;
            // a resident block's buffers are freed for the next channel block only
            const bool release = !resident || (after < run.end && run.block_of(after) != run.n0);
            const int pairs = run.nz / 2 + 1 + (run.nz & 1);
            RollRing done = slot;                           // the pair that the last slice completes next
            for (int sl = 0; sl < slices && !fault; ++sl) {
                if (!warp_wait(wfull0 + 8 * wr.i, wr.phase)) {
                    fault = true;
                    break;
                }
                const uint64_t bd0 = umma_desc_sw32(sw + wr.i * S::WSLICE, 256);
                int s0 = 2 * slot.i;                        // the slot of output plane 2 p of halo pair p
                for (int p = 0; p < pairs; ++p) {
                    if (!warp_wait(full0 + 8 * st.i, st.phase)) {
                        fault = true;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const uint64_t ad2 = umma_desc_sw32(sh + st.i * S::STAGE, S::HX * 32);
#pragma unroll
                    for (int zz = 0; zz < 2; ++zz) {
                        // halo plane i reaches planes hi, hi - 1, .. lo through taps dz0, dz0 + 1, ..: ascending
                        // columns up to the ring's end (n1 of them), the rest from column 0
                        const int i = 2 * p + zz, hi = min(i, run.nz - 1), lo = max(i - 2, 0), cnt = hi - lo + 1, dz0 = i - hi;
                        if (cnt <= 0) continue;             // past the last halo plane of an odd piece
                        int s = s0 + zz - dz0;              // the slot of plane hi
                        if (s < 0) s += R;
                        const int n1 = min(cnt, s + 1), n2 = cnt - n1;
                        const uint32_t d1 = tmem + (uint32_t)((R - 1 - s) * BN);
                        const uint64_t ad0 = ad2 + (uint64_t)(zz * S::ZPLANE / 16);
                        const uint64_t bd = bd0 + (uint64_t)(2 * dz0 * BN);
                        const uint32_t id1 = umma_idesc_bf16(n1 * BN);
#pragma unroll
                        for (int t = 0; t < 9; ++t)
                            umma_f16(lead, d1, ad0 + (uint64_t)(2 * ((t / 3) * S::HX + t % 3)), bd + (uint64_t)(2 * t * S::N3), id1, 1u);
                        if (n2 > 0) {
                            const uint64_t b2 = bd + (uint64_t)(2 * n1 * BN);
                            const uint32_t id2 = umma_idesc_bf16(n2 * BN);
#pragma unroll
                            for (int t = 0; t < 9; ++t)
                                umma_f16(lead, tmem, ad0 + (uint64_t)(2 * ((t / 3) * S::HX + t % 3)), b2 + (uint64_t)(2 * t * S::N3), id2, 1u);
                        }
                    }
                    umma_commit(lead, empty0 + 8 * st.i);
                    st.step();
                    s0 = s0 + 2 == R ? 0 : s0 + 2;
                    if (sl == slices - 1 && p > 0) {
                        umma_commit(lead, pfull0 + 8 * done.i);
                        done.step();
                    }
                }
                if (release) umma_commit(lead, wempty0 + 8 * wr.i);
                wr.step();
            }
            slot = done;
        }
        // the last release comes behind the commits that the epilogue waits for: it arrives before the CTA ends
        if (!resident && !fault) fault = !warp_wait(wempty0 + 8 * ((wr.i == 0 ? wbufs : wr.i) - 1), wr.phase ^ (wr.i == 0 ? 1u : 0u));
    } else {
        // ---- epilogue: warps 0-3 and 4-7 take turns at pairs of planes ------------------------------------
        const int wg = warp >> 2, r = (warp & 3) * 32 + lane;       // accumulator row = TMEM lane = voxel of a plane
        const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        RollRing slot(RP);
        int turn = 0;
        float bs[BN];
        while (!fault && run.next()) {
#pragma unroll
            for (int c = 0; c < BN; ++c) bs[c] = bias ? bias[run.n0 + c] : 0.f;
            const int yy = run.y0 + (r >> 3), xx = run.x0 + (r & 7);
            const bool in = yy < g.h && xx < g.w;
            const long long hw = (long long)g.h * g.w;
            const long long v0 = ((long long)run.n * g.d + run.z0) * hw + (long long)yy * g.w + xx;
            for (int o = 0; o < run.nz; o += 2, slot.step(), turn ^= 1) {
                if (turn != wg) continue;
                if (!warp_wait(pfull0 + 8 * slot.i, slot.phase)) {
                    fault = true;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
                for (int zz = 0; zz < 2; ++zz) {
                    const uint32_t col = trow + (uint32_t)((R - 1 - (2 * slot.i + zz)) * BN);
                    uint32_t v[BN];
#pragma unroll
                    for (int c0 = 0; c0 < BN; c0 += 16) tmem_ld16(col + c0, *reinterpret_cast<uint32_t(*)[16]>(&v[c0]));
#pragma unroll
                    for (int c0 = 0; c0 < BN; c0 += 16) tmem_zero16(col + c0);
                    if (zz == 1) {
                        tmem_store_wait();
                        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                        __syncwarp();
                        if (lane == 0) mbar_arrive(pempty0 + 8 * slot.i);
                    }
                    if (in && o + zz < run.nz) {
                        const long long at = (v0 + (o + zz) * hw) * cout + run.n0;
                        // the mask of up to 48 channels before their first store, which it must not wait for
                        constexpr int MB = BN > 48 ? BN / 2 : BN;
#pragma unroll
                        for (int b = 0; b < BN; b += MB) {
                            uint32_t mk[MB / 2];
                            if (mask) {
#pragma unroll
                                for (int c0 = 0; c0 < MB; c0 += 16) roll_mask16(mask + at + b + c0, mk + c0 / 2);
                            }
#pragma unroll
                            for (int c0 = 0; c0 < MB; c0 += 16)
                                roll_store16(v + b + c0, bs + b + c0, mask ? mk + c0 / 2 : nullptr, y + at + b + c0, relu, wide != 0);
                        }
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
