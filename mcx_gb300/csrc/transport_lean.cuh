// transport_lean.cuh -- the transport kernel of the plain path: label media, per-photon streams,
// flux / fluence / energy into an FP32 field, no roulette, every photon scattering with its own g
// (lean_path() in transport.cu is the rule).  Included by transport.cu inside its namespace.
//
// Photon for photon the arithmetic is transport_kernel's (the same draws, the same operations in
// the same order on position, direction, weight, time and scattering length), so both give the
// same paths, records and counters bit for bit; the fluence differs by the order of its sums.  What
// differs is how much is issued around that arithmetic.  transport_kernel issued 16 warp
// instructions per photon step (272 per lane-step at 17 lanes) at 87% of the issue slots: it is
// bound by issue, and a lone photon by the length of its step.  Here
//   * switches that a launch fixes (seeding scheme, roulette, field type, gscatter, saved output)
//     are resolved by choosing this kernel and cost nothing per step;
//   * a step ends in its voxel (and scatters), or crosses into a voxel of the same medium, or is an
//     event (another medium, the outside, the end of the window); only events run the boundary,
//     detector, reflection and termination rules, and only an event reloads medium properties;
//   * the divisions by a medium's mus and mua are products with reciprocals taken once per launch by
//     the same instruction, and the absorbed weight of a photon is a difference taken at its end;
//   * the label of the voxel entered is requested before the deposit and the scattering of the
//     warp's other lanes and looked at after them;
//   * conditions on the way are evaluated without short cuts and the crossed axis by selection:
//     branches there ran three versions of the crossing for a few lanes each (13 lanes per
//     instruction; 44.5 against 37.1 ms on the sphere deck at 8e6 photons).
//   * truth values do not outlive a branch: seven predicates do not hold them, and packing and unpacking
//     them cost 12 of 179 thread instructions a step (17.1 -> 16.5 ms on the cube at 8e6 photons).
// Measured, kernel time in transport_kernel and here (GB300, 2070 MHz): sphere with 50 gates and four
// detectors, 2e6 photons, 18.4 -> 11.8 ms; layered 128^3 head, 3e5, 43.3 -> 18.7; planar source, 1e6, 9.24 ->
// 5.20; homogeneous cube, 2e6, 7.96 -> 5.42 and 1e4 photons, 2.84 -> 1.23.  On the cube 167 thread instructions
// a step instead of 223, 16 lanes an instruction, 83% of the issue slots: what binds it is issue still, the
// scattering and the crossing block each run by the half of the lanes that need it.
//
// REPLAY runs detected photons again from their saved states into the Jacobian of absorption (or its time-of-flight
// weighted form).  A replay has about a photon a thread, so it lasts as long as its longest photon, and that as its steps:
// 44 829 photons of the reflecting cube took 5.5 ms in transport_kernel's variant with every replay option and 1.46
// here; with two media, a void pocket and reflection 6.0 and 1.65.

constexpr int kLeanBlock = 256, kLeanWarps = kLeanBlock / 32;

// Shared memory of a CTA.  Everything but the record accumulators and the tile lies at offsets fixed
// at compile time (thread arrays have room for the largest block), so an access is one instruction
// on a thread's own address instead of a sum of launch parameters.
struct LeanSmem {
    float4 prop[kMaxMedia];                     // (mua, mus, g, n)
    float2 inv[kMaxMedia];                      // (1 / mus, deposit per absorbed weight)
    unsigned long long pool[2 * kLeanWarps];    // per warp: next, end of its photon-index pool
    ulonglong2 queue[kLeanBlock];               // per warp: the random states of photons drawn ahead,
    float qscat[kLeanBlock];                    // and their first scattering lengths
    unsigned wcount[2 * kLeanWarps];            // per warp: launches tried, photons run
    unsigned steps[kLeanBlock];                 // steps of the photons the lane has finished
    unsigned nscat0[kLeanBlock];                // detector runs: the lane's scatter count at the last change of medium
    float wlaunch[kLeanBlock];                  // launch weight of its photon
    float tally[kNumEnergy * kLeanBlock];       // FP32 per-thread partial sums
    float ppath[1];                             // partialdata x kLeanBlock (detector runs), then the tile
};

inline size_t lean_smem_bytes(const KParams& p, bool savedet, bool tile) {
    size_t b = offsetof(LeanSmem, ppath);
    if (savedet) b += sizeof(float) * (size_t)p.partialdata * kLeanBlock;
    if (tile) b += sizeof(unsigned) * (size_t)p.tnx * p.tny * p.tnz * p.tng;
    return b;
}

// transmit() with the roundings the compiler gives it in transport_kernel spelt out: left to itself it fuses the sums of
// squares one way or the other by what surrounds them, and the photons part.
__device__ __forceinline__ void transmit_as_general(float& vx, float& vy, float& vz, float n1, float n2, int axis) {
    const float r = __fdividef(n1, n2);
    vx = __fmul_rn(vx, r); vy = __fmul_rn(vy, r); vz = __fmul_rn(vz, r);
    const float a = axis == 0 ? vy : vx, b = axis == 2 ? vy : vz, v = axis == 0 ? vx : (axis == 1 ? vy : vz);
    const float s = __fmaf_rn(a, a, __fmul_rn(b, b));
    const float q = (s < 1.f) ? sqrtf(__fsub_rn(1.f, s)) * (float)((v > 0.f) - (v < 0.f)) : 0.f;
    vx = axis == 0 ? q : vx;
    vy = axis == 1 ? q : vy;
    vz = axis == 2 ? q : vz;
    const float k = rsqrtf(__fmaf_rn(vz, vz, __fmaf_rn(vy, vy, __fmul_rn(vx, vx))));
    vx = __fmul_rn(vx, k); vy = __fmul_rn(vy, k); vz = __fmul_rn(vz, k);
}

constexpr unsigned kOutside = 0xFFFFFFFFu;      // no voxel's index: a volume has fewer than 2^32 - 1 voxels

__device__ __forceinline__ float ahead(float v) { return v > 0.f ? 1.f : 0.f; }

// A warp launches its lanes anew when this many are out of photons.  Sampling an area source and walking its photon
// through the void is long, and run for one lane it holds 31: four at a time took the planar source from 14.2 to
// 11.7 ms at 3e6 photons (2: 13.1, 3: 12.0, 6: 11.8, 8: 11.9).  A pencil's launch is short: waiting for a second
// lane costs what it saves (16.9 -> 17.1 ms on the cube at 8e6).
template <bool AREA>
constexpr unsigned kLeanTogether = AREA ? 4u : 1u;

// What a launch of the kernel is for: at least four photons a thread; fewer, spread over all warps where they are fewer than
// its lanes (in the same kernel the spare lanes' arithmetic cost the long runs 1%); a replay.
enum LeanKind : int { kLeanMany = 0, kLeanFew, kLeanReplays };

template <bool REFLECT, bool SAVEDET, bool AREA, int KIND, int MINB>
__global__ void __launch_bounds__(kLeanBlock, MINB) lean_kernel(const __grid_constant__ KParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    LeanSmem& S = *reinterpret_cast<LeanSmem*>(smem_raw);
    constexpr unsigned B = kLeanBlock, kTogether = kLeanTogether<AREA>;
    constexpr bool REPLAY = KIND == kLeanReplays, QUEUE = KIND == kLeanMany && !AREA && !SAVEDET && !REFLECT;
    const unsigned spare = KIND == kLeanMany ? 0u : P.spare;        // lanes left without a photon
    unsigned* const tile = reinterpret_cast<unsigned*>(S.ppath) + (SAVEDET ? P.partialdata * B : 0u);
    const unsigned tid = threadIdx.x;
    const unsigned lane = tid & 31u;
    const unsigned warp = tid >> 5;

    for (unsigned i = tid; i < (unsigned)P.medianum; i += blockDim.x) {
        const float4 m = P.prop[i];
        S.prop[i] = m;
        // the deposit per absorbed weight: 1 / mua, 1 for the energy output, negative where the
        // deposit is the path instead (a medium that does not absorb)
        const float per = (P.outputtype == kOutEnergy) ? 1.f : (m.x < kEPS) ? -1.f : __fdividef(1.f, m.x);
        S.inv[i] = make_float2(__fdividef(1.f, m.y), per);
    }
    for (int k = 0; k < kNumEnergy; k++) S.tally[k * B + tid] = 0.f;
    const int tile_elems = P.tile_on ? P.tnx * P.tny * P.tnz * P.tng : 0;
    for (int i = tid; i < tile_elems; i += blockDim.x) tile[i] = 0u;
    if (lane == 0) {
        S.pool[2 * warp] = 0ull;
        S.pool[2 * warp + 1] = 0ull;
        S.wcount[2 * warp] = 0u;
        S.wcount[2 * warp + 1] = 0u;
    }
    __syncthreads();

    bool alive = false, ended = false;  // ended: its photon has ended and is not accounted for yet
    unsigned fate = 0u;                 // how, for the detectors: the reference's detector flag
    // warp-uniform: dead lanes that make the warp draw photons; out of reach when there are none left
    constexpr unsigned kNever = 64u;
    unsigned refill_at = P.src_ok == 0 ? kNever : kTogether + spare;
    float px = 0.f, py = 0.f, pz = 0.f, vx = 0.f, vy = 0.f, vz = 1.f, rvx = 0.f, rvy = 0.f, rvz = 0.f;
    float fx = 0.f, fy = 0.f, fz = 0.f; // integer coordinates of the current voxel, as floats
    float w = 0.f, w0 = 0.f, t = 0.f, pscat = 0.f, pathlen = 0.f, segp = 0.f;
    float mua = 0.f, mus = 0.f, n = 1.f, rmus = 0.f, rmua = 0.f;      // the current medium
    // index the next face sees on this side: transport_kernel's pr.w at the end of the step before
    float n1 = 1.f;
    unsigned idx = 0u;
    unsigned lab = 0u;                  // label byte of the current voxel
    // bit 7: the reference's detector flag at the end of the step before -- the current voxel's, or
    // after a reflection the voxel's bounced off, until the photon scatters
    unsigned carry = 0u;
    unsigned long long r0 = 0ull, r1 = 0ull;
    float eabs = 0.f;                   // absorbed weight of the photon recorded in the field
    unsigned left = 0u;                 // steps the photon may still take
    float rw = 0.f, rtof = 1.f;         // replay: detected weight, time of flight where the output carries it
    int rbin = -1;                      // replay: its field block (gate + detector offset), -1 none
    unsigned c_scat = 0u, c_dep = 0u, c_tile = 0u;
    S.steps[tid] = 0u;
    unsigned q_next = 0u, q_left = 0u;  // warp-uniform: photons drawn ahead
    // the step cap ends a photon 1023 steps past it, the latest transport_kernel does
    const unsigned limit = P.step_cap < 0xFFFFFC00u ? P.step_cap + 1023u : 0xFFFFFFFFu;

    // The end of a photon: detection and energy bookkeeping (src/mcx_core.cu:1113-1182, 365-417)
    const auto finish = [&]() {
        ended = false;
        bool detected = false;
        if (SAVEDET && (fate & kDET_MASK)) {
            const int detid = (fate == kOUT_MIN) ? -1 : find_detector(P, px, py, pz);
            if (detid) {
                detected = true;
                const unsigned slot = atomicAdd(P.detcount, 1u);
                if (slot < P.maxdet) {
                    float* rec = P.detp + (size_t)slot * P.reclen;
                    unsigned k = 0;
                    if (P.savedetflag & 0x1u) rec[k++] = (float)detid;
                    for (unsigned i = 0; i < P.partialdata; i++) rec[k++] = S.ppath[i * B + tid];
                    if (P.savedetflag & 0x10u) { rec[k++] = px; rec[k++] = py; rec[k++] = pz; }
                    if (P.savedetflag & 0x20u) { rec[k++] = vx; rec[k++] = vy; rec[k++] = vz; }
                    if (P.savedetflag & 0x40u) rec[k++] = S.wlaunch[tid];
                }
            }
        }
        S.tally[kELaunch * B + tid] += S.wlaunch[tid];
        S.tally[(detected ? kEDetect : kEEscape) * B + tid] += w;
        S.tally[kEAbsDep * B + tid] += eabs;
        S.tally[kEAbsOther * B + tid] += (S.wlaunch[tid] - w) - eabs;
        S.steps[tid] += limit - left;
        if (left == 0u) atomicOr(P.errflag, kErrStepCap);
    };

    while (true) {
        // ---- relaunch lanes that have no photon (warp-uniform control flow) ------------------
        const unsigned live = __ballot_sync(kFull, alive);
        if (live != kFull) {
            const unsigned idle = __popc(~live);
            if (!live || idle >= refill_at) {
                if (AREA && ended) finish();
                if (refill_at == kNever) break;
                const unsigned want = ~live;
                const unsigned cnt = idle - spare;
                const unsigned rank = __popc(want & ((1u << lane) - 1u));
                bool start;
                float first = 0.f;
                if constexpr (QUEUE) {
                    // A lane of a pencil's warp dies every six steps or so, and all wait for its relaunch: the seeding and
                    // the first flight are drawn for up to 32 photons at a time, a lane each (cube, 8e6 photons 16.5 ->
                    // 15.9 ms, 1e6 3.66 -> 3.60).  Not with an area source, whose kernel spills more with it (26.9 -> 27.2
                    // on the planar source at 8e6), nor with detector records (two media, 3e5: 4.05 -> 4.14) or reflection
                    // (layered head, 1e6: 25.0 -> 25.5), where a photon lives longer and the registers are fewer.
                    if (q_left == 0u) {
                        const unsigned take = max(cnt, P.ahead);
                        unsigned long long base = 0ull;
                        if (lane == 0) base = atomicAdd(P.work, (unsigned long long)take);
                        base = __shfl_sync(kFull, base, 0);
                        __syncwarp();           // every lane has read the entries before that are overwritten here
                        if (lane < take && base + lane < P.d_nwork) {
                            ulonglong2 q;
                            seed_photon(P.seed, P.photon_offset + base + lane, q.x, q.y);
                            // the launch flight takes the first of its step's three numbers
                            float u_len, u_phi, u_th;
                            rng_next3(q.x, q.y, u_len, u_phi, u_th);
                            S.qscat[tid] = -__logf(u_len + kEPS);
                            S.queue[tid] = q;
                        }
                        q_next = tid - lane;
                        q_left = base >= P.d_nwork ? 0u : (unsigned)min((unsigned long long)take, P.d_nwork - base);
                        if (q_left == 0u) refill_at = kNever;
                        __syncwarp();           // and reads the new ones after they are written
                    }
                    start = !alive && rank < q_left;
                    if (start) {
                        const ulonglong2 q = S.queue[q_next + rank];
                        r0 = q.x;
                        r1 = q.y;
                        first = S.qscat[q_next + rank];
                    }
                    const unsigned taken = min(cnt, q_left);
                    q_next += taken;
                    q_left -= taken;
                } else {
                    unsigned long long pool_next = S.pool[2 * warp], pool_end = S.pool[2 * warp + 1];
                    const unsigned long long avail = pool_end - pool_next;
                    unsigned long long mine = pool_next + rank;
                    if (avail < cnt) {
                        // reserve at least what the dead lanes need, normally a whole chunk
                        const unsigned long long take = max((unsigned long long)P.chunk, (unsigned long long)(cnt - avail));
                        unsigned long long base = 0ull;
                        if (lane == 0) base = atomicAdd(P.work, take);
                        base = __shfl_sync(kFull, base, 0);
                        if (rank >= avail) mine = base + (rank - avail);
                        pool_next = base + (cnt - avail);
                        pool_end = base + take;
                        if (base >= P.d_nwork) refill_at = kNever;
                    } else {
                        pool_next += cnt;
                    }
                    __syncwarp();               // every lane has read the pool before lane 0 rewrites it
                    if (lane == 0) {
                        S.pool[2 * warp] = pool_next;
                        S.pool[2 * warp + 1] = pool_end;
                    }
                    __syncwarp();               // and reads the new one at the next refill
                    start = !alive && mine < P.d_nwork && (KIND == kLeanMany || rank < cnt);
                    if (start) {
                        if constexpr (REPLAY) {
                            // a detected photon again: its saved launch state and detection record
                            // (src/mcx_core.cu:1203-1211)
                            r0 = __ldg(P.replay_seed + 2 * mine);
                            r1 = __ldg(P.replay_seed + 2 * mine + 1);
                            const float tof = __ldg(P.replay_tof + mine);
                            rbin = (int)floorf((tof - P.twin0) * P.Rtstep);
                            if (rbin < 0 || rbin >= P.maxgate) rbin = -1;      // detected outside this gate group
                            else if (P.replaydet == -1) rbin += ((__ldg(P.replay_detid + mine) & 0xFFFF) - 1) * P.maxgate;
                            rw = __ldg(P.replay_w + mine);
                            if (P.outputtype == kOutWLTOF) rtof = tof;
                            // the draw by which the recorded run picked its source (src/mcx_core.cu:1229-1231)
                            if (P.srcid >= 1) (void)rng_next(r0, r1);
                        } else {
                            seed_photon(P.seed, P.photon_offset + mine, r0, r1);
                        }
                    }
                }
                bool entered = false;
                if (start) {
                    if (!AREA || P.srctype == kSrcPencil) {
                        // the pencil's launch state, traced through the void by the host
                        px = P.src_p.x; py = P.src_p.y; pz = P.src_p.z; w = P.src_p.w;
                        vx = P.src_v.x; vy = P.src_v.y; vz = P.src_v.z;
                        t = P.src_t * P.d_inv_c0;
                        idx = P.src_idx;
                        lab = P.src_label;
                        fx = (float)P.src_fx; fy = (float)P.src_fy; fz = (float)P.src_fz;
                        entered = true;
                    } else if constexpr (AREA) {
                        Launch L;
                        entered = launch_source<false, false>(P, r0, r1, L);
                        if (entered) {
                            px = L.px; py = L.py; pz = L.pz; w = L.w;
                            vx = L.vx; vy = L.vy; vz = L.vz;
                            t = L.t;
                            idx = L.idx;
                            lab = L.label;
                            fx = (float)L.ix; fy = (float)L.iy; fz = (float)L.iz;
                        }
                    }
                    if (entered) {
                        rvx = __fdividef(1.f, vx); rvy = __fdividef(1.f, vy); rvz = __fdividef(1.f, vz);
                        carry = lab;
                        const float4 pr = S.prop[lab & kLabelMask];
                        const float2 iv = S.inv[lab & kLabelMask];
                        mua = pr.x; mus = pr.y; n = pr.w; n1 = pr.w;
                        rmus = iv.x; rmua = iv.y;
                        if (QUEUE) {
                            pscat = first;
                        } else {
                            // the launch flight takes the first of its step's three numbers
                            float u_len, u_phi, u_th;
                            rng_next3(r0, r1, u_len, u_phi, u_th);
                            pscat = -__logf(u_len + kEPS);
                        }
                        S.wlaunch[tid] = w;
                        w0 = w;
                        eabs = 0.f;
                        left = limit;
                        pathlen = 0.f;
                        if (SAVEDET) {
                            segp = 0.f;
                            S.nscat0[tid] = c_scat;
                            for (unsigned k = 0; k < P.partialdata; k++) S.ppath[k * B + tid] = 0.f;
                        }
                        alive = true;
                    }
                }
                const unsigned attempted = __ballot_sync(kFull, start), ran = __ballot_sync(kFull, entered);
                if (lane == 0) {
                    S.wcount[2 * warp] += __popc(attempted);
                    S.wcount[2 * warp + 1] += __popc(ran);
                }
                if (!__any_sync(kFull, alive)) {
                    if (attempted == 0u) break;     // no photon left for any lane of this warp
                    continue;
                }
            }
        }
        if (!alive) continue;

        // ---- one step (src/mcx_core.cu:1888-2514) --------------------------------------------
        // distance to the nearest voxel face (hitgrid, src/mcx_core.cu:493-507)
        const float hx = fabsf((fx + ahead(vx) - px) * rvx);
        const float hy = fabsf((fy + ahead(vy) - py) * rvy);
        const float hz = fabsf((fz + ahead(vz) - pz) * rvz);
        const float dist = fminf(fminf(hx, hy), hz);
        // src/mcx_core.cu:2101-2109
        const float sdist = dist * mus;
        const bool cross = sdist < pscat;                   // else the flight ends inside this voxel
        const float slen = cross ? sdist : pscat;
        const float len = cross ? dist : pscat * rmus;
        px = fmaf(len, vx, px);
        py = fmaf(len, vy, py);
        pz = fmaf(len, vz, pz);
        w *= __expf(-mua * len);                                        // 2140
        pscat -= slen;
        t = fmaf(len, n, t);                                            // t += len*n/c0, in grid units
        pathlen += len;
        left--;

        // What the event below needs of a crossing is kept as numbers it compares again: truth values that live
        // past a branch are packed into registers and unpacked at every step.
        unsigned labn = lab, idxn = idx;        // idxn: kOutside where the photon leaves the volume
        float fn = 0.f;
        if (cross) {
            // The face crossed, by selection: a branch per axis would run each of the three for its own lanes.
            const bool ax = dist == hx, ay = !ax & (dist == hy);
            // only the crossed axis can leave the volume (2169-2186)
            const float va = ax ? vx : (ay ? vy : vz);
            const float fa = ax ? fx : (ay ? fy : fz);
            const float la = ax ? P.d_fnx : (ay ? P.d_fny : P.d_fnz);
            const unsigned stride = ax ? 1u : (ay ? (unsigned)P.nx : P.dimxy);
            const bool up = va > 0.f;
            idxn = up ? idx + stride : idx - stride;
            fn = fa + (up ? 1.f : -1.f);
            const bool valid = (fn >= 0.f) & (fn < la) & (idxn < P.nvox);
            labn = (unsigned)__ldg(P.labels + (valid ? idxn : idx));
            idxn = valid ? idxn : kOutside;

            // deposit into the voxel just left, time bin taken at exit (2191-2292)
            const float dw = w0 - w;
            float weight = (rmua < 0.f) ? (w0 * pathlen) : dw * rmua;
            if (REPLAY) weight = (rbin < 0) ? 0.f : rw * pathlen * rtof;        // mua Jacobian (x time of flight)
            const bool rec = (t >= P.d_tw0) & (t < P.d_tw1) & (weight != 0.f);
            eabs += rec ? dw : 0.f;
            c_dep += rec;
            // (a deposit that passed the window test may compute bin -1 at a window that does not
            // start at 0: it belongs to the first gate)
            int tshift = 0;
            if (REPLAY) tshift = rbin;
            else if (P.maxgate > 1) tshift = min(P.maxgate - 1, max(0, (int)floorf(fmaf(t, P.d_bin_a, -P.d_bin_b))));
            float* const slot = P.field + ((size_t)tshift * P.nvox + idx);
            // the index range of the tile box (empty without a tile) screens most deposits out
            // with one compare before the box test
            bool in_tile = false;
            if (!REPLAY && idx - P.d_tile_lo < P.d_tile_span) {
                const float ox = fx - P.d_tx0, oy = fy - P.d_ty0, oz = fz - P.d_tz0;
                in_tile = (ox >= 0.f) & (ox < P.d_tnx) & (oy >= 0.f) & (oy < P.d_tny) & (oz >= 0.f) & (oz < P.d_tnz) &
                          rec & (weight > 0.f) & ((unsigned)(tshift - P.tg0) < (unsigned)P.tng);
                if (in_tile) {
                    // exact in FP32: a tile has fewer than 2^24 slots
                    const unsigned ti = (unsigned)fmaf(fmaf(fmaf((float)(tshift - P.tg0), P.d_tnz, oz), P.d_tny, oy), P.d_tnx, ox);
                    // exact fixed-point sum (see transport_kernel)
                    const unsigned q = __float_as_uint(fmaf(weight, P.d_tile_scale, 8388608.f)) - 0x4B000000u;
                    const unsigned old = atomicAdd(tile + ti, q);
                    if ((old < kTileFlushUnits) & (old + q >= kTileFlushUnits)) {
                        atomicSub(tile + ti, kTileFlushUnits);
                        field_add_large(P, slot - P.field, P.d_tile_flush);
                    }
                    c_tile++;
                }
            }
            if (rec & !in_tile) atomicAdd(slot, weight);
            w0 = w;
            if (SAVEDET) segp += pathlen;
            pathlen = 0.f;
            fx = ax ? fn : fx;
            fy = ay ? fn : fy;
            fz = (ax | ay) ? fz : fn;
        } else if (!((t > P.d_tw1) | (left == 0u))) {
            // ---- scattering event: random numbers in MCX's order (scattering length, azimuth,
            // zenith), one generator step for all three
            float u_len, u_phi, u_th;
            rng_next3(r0, r1, u_len, u_phi, u_th);
            pscat = -__logf(u_len + kEPS);                              // src/mcx_rand_xorshift128p.cu:122
            float sphi, cphi;
            __sincosf(kTWO_PI * u_phi, &sphi, &cphi);                   // src/mcx_core.cu:1930-1933
            const float g = S.prop[lab & kLabelMask].z;
            // Henyey-Greenstein (1946-1959), isotropic where g is 0 (1961-1963)
            const float g2 = g * g;
            float tmp = __fdividef(1.f - g2, 1.f - g + 2.f * g * u_th);
            tmp *= tmp;
            float ct = __fdividef(1.f + g2 - tmp, 2.f * g);
            ct = fmaxf(-1.f, fminf(1.f, ct));
            ct = (fabsf(g) > kEPS) ? ct : 2.f * u_th - 1.f;
            const float st = sqrtf(fmaxf(0.f, 1.f - ct * ct));
            if (SAVEDET && ((P.savedetflag >> 3) & 1u) && (lab & kLabelMask)) {     // momentum transfer, 1970-1993
                const unsigned fS = (P.savedetflag >> 1) & 1u, fP = (P.savedetflag >> 2) & 1u;
                S.ppath[((unsigned)P.nmedia_det * (fS + fP) + (lab & kLabelMask) - 1u) * B + tid] += 1.f - ct;
            }
            rotate(vx, vy, vz, st, ct, sphi, cphi);
            rvx = __fdividef(1.f, vx); rvy = __fdividef(1.f, vy); rvz = __fdividef(1.f, vz);
            c_scat++;
            if (SAVEDET) carry = lab;
        }

        bool kill = (t > P.d_tw1) | (left == 0u);
        if (!kill & (idxn != kOutside) & (((labn ^ lab) & kLabelMask) == 0u)) {
            // the same medium: nothing else to do
            idx = idxn;
            lab = labn;
            if (SAVEDET) carry = labn;
            if (REFLECT) n1 = n;
            continue;
        }

        // ---- event: another medium, the outside, the end of the window or the step cap ----------
        const int axis = (dist == hx) ? 0 : ((dist == hy) ? 1 : 2);
        const bool valid = idxn != kOutside;
        const unsigned idxold = idx, medold = lab & kLabelMask;
        const unsigned detold = (carry & kLabelDet) ? kDET_MASK : 0u;   // mediaidold's detector bit (2167)
        unsigned med = medold;
        unsigned detflag = 0u;
        int bcf = BC_UNKNOWN;
        const bool outmax = !(fn < 0.f);
        float nstart = n;               // the side the next face sees, unless the photon refracts
        if (cross) {
            if (valid) {
                med = labn & kLabelMask;
                idx = idxn;
                carry = labn;
            } else {
                // the voxel index has lost step with the coordinates: never read or write out of
                // the volume; the photon leaves and the host reports the error
                if (fn >= 0.f && fn < ((axis == 0) ? P.d_fnx : ((axis == 1) ? P.d_fny : P.d_fnz))) atomicOr(P.errflag, kErrIndex);
                med = 0u;
                bcf = P.bc[(outmax ? 3 : 0) + axis];
                carry = 0u;             // a boundary code, never the detector bit
            }
            // leaving into a 0 voxel or the outside without reflection (2307-2354)
            if (med == 0u && ((!REFLECT || n1 == P.d_n0) || (bcf == BC_UNKNOWN && !P.doreflect) || bcf == BC_ABSORB ||
                              bcf == BC_CYCLIC) && bcf != BC_MIRROR)
                kill = true;
        }
        bool wrapped = false;
        // (never for the step cap: on a periodic axis one voxel thick every step ends here)
        if (kill && left != 0u && !valid && bcf == BC_CYCLIC) {         // 2311-2335
            const float span = (axis == 0) ? P.d_fnx : ((axis == 1) ? P.d_fny : P.d_fnz);
            const float shift = outmax ? -span : span;
            if (axis == 0) { px = nextafter_mcx(roundf(px + shift), (vx > 0.f) - (vx < 0.f), P.maxvoidstep); fx = floorf(px); }
            else if (axis == 1) { py = nextafter_mcx(roundf(py + shift), (vy > 0.f) - (vy < 0.f), P.maxvoidstep); fy = floorf(py); }
            else { pz = nextafter_mcx(roundf(pz + shift), (vz > 0.f) - (vz < 0.f), P.maxvoidstep); fz = floorf(pz); }
            if (fx >= 0.f && fx < P.d_fnx && fy >= 0.f && fy < P.d_fny && fz >= 0.f && fz < P.d_fnz) {
                idx = (unsigned)fz * P.dimxy + (unsigned)fy * (unsigned)P.nx + (unsigned)fx;
                labn = (unsigned)__ldg(P.labels + idx);
                med = labn & kLabelMask;
                carry = labn;
                kill = false;
                wrapped = true;
            }
        }
        if (kill) {
            detflag = (!valid && P.bc[(outmax ? 9 : 6) + axis]) ? kOUT_MIN : detold;
        } else if (REFLECT && cross && !wrapped) {
            // Fresnel reflection / refraction on crossing (2381-2503)
            const float n2 = S.prop[med].w;
            if (((med && P.doreflect) ||
                 (med == 0u && ((bcf == BC_UNKNOWN && P.doreflect) || bcf == BC_REFLECT || bcf == BC_MIRROR))) &&
                (bcf == BC_MIRROR || n1 != n2)) {
                float Rtotal = 1.f;
                const float a2 = n1 * n1, b2 = n2 * n2;
                const float va = (axis == 0) ? vx : ((axis == 1) ? vy : vz);
                const float cphi = fabsf(va);
                const float sphi = 1.f - cphi * cphi;
                const float c2 = 1.f - __fdividef(a2, b2) * sphi;
                if (c2 > 0.f && bcf != BC_MIRROR) {
                    float ctheta = a2 * cphi * cphi + b2 * c2;
                    const float stheta = 2.f * n1 * n2 * cphi * sqrtf(c2);
                    Rtotal = __fdividef(ctheta - stheta, ctheta + stheta);
                    ctheta = b2 * cphi * cphi + a2 * c2;
                    Rtotal = (Rtotal + __fdividef(ctheta - stheta, ctheta + stheta)) * 0.5f;
                }
                if (Rtotal < 1.f && !(med == 0u && bcf == BC_MIRROR) && rng_next(r0, r1) > Rtotal) {
                    transmit_as_general(vx, vy, vz, n1, n2, axis);
                    if (med == 0u) {
                        kill = true;
                        detflag = (!valid && P.bc[(outmax ? 9 : 6) + axis]) ? kOUT_MIN : detold;
                    } else {
                        nstart = n2;
                    }
                } else {
                    // mirror the direction and nudge the position back into the voxel left
                    if (axis == 0) {
                        vx = -vx;
                        px = nextafter_mcx(rintf(px), (vx > 0.f) - (vx < 0.f), P.maxvoidstep);
                        fx = floorf(px);
                    } else if (axis == 1) {
                        vy = -vy;
                        py = nextafter_mcx(rintf(py), (vy > 0.f) - (vy < 0.f), P.maxvoidstep);
                        fy = floorf(py);
                    } else {
                        vz = -vz;
                        pz = nextafter_mcx(rintf(pz), (vz > 0.f) - (vz < 0.f), P.maxvoidstep);
                        fz = floorf(pz);
                    }
                    idx = idxold;
                    med = medold;
                    labn = lab;                 // carry keeps the bounced-off value
                }
                rvx = __fdividef(1.f, vx); rvy = __fdividef(1.f, vy); rvz = __fdividef(1.f, vz);
            }
        }

        if (SAVEDET && (kill || med != medold)) {
            // per-medium partial path and scattering count of the segment that ends (1970-1981, 2152-2165)
            segp += pathlen;        // the last voxel's path when the photon ends inside it, else 0
            if (medold > 0u) {
                const unsigned fS = (P.savedetflag >> 1) & 1u, fP = (P.savedetflag >> 2) & 1u;
                if (fS) S.ppath[(medold - 1u) * B + tid] += (float)(c_scat - S.nscat0[tid]);
                if (fP) S.ppath[((unsigned)P.nmedia_det * fS + (medold - 1u)) * B + tid] += segp;
            }
            S.nscat0[tid] = c_scat;
            segp = 0.f;
        }
        if (!kill) {
            lab = valid || wrapped ? labn : lab;
            n1 = nstart;
            if (!valid && !wrapped && med != medold) {
                // outside the volume without ending or being turned back: the background's row, as
                // transport_kernel gives it; its next crossing finds the index out of the volume
                lab = 0u;
                idx = outmax ? kOUT_MAX : kOUT_MIN;
            }
            const float4 pr = S.prop[med];
            const float2 iv = S.inv[med];
            mua = pr.x; mus = pr.y; n = pr.w;
            rmus = iv.x; rmua = iv.y;
            continue;
        }
        // the photon ends (an area source's lane keeps its last state until its warp launches some together)
        alive = false;
        ended = true;
        fate = (SAVEDET && med == 0u) ? detflag : 0u;
        if (!AREA) finish();
    }

    // ---- flush: tile, tallies, counters ------------------------------------------------------
    __syncthreads();
    for (int i = tid; i < tile_elems; i += blockDim.x) {
        const unsigned q = tile[i];
        if (q == 0u) continue;
        const float v = (float)((double)q / (double)P.d_tile_scale);
        int r = i;
        const int x = r % P.tnx; r /= P.tnx;
        const int y = r % P.tny; r /= P.tny;
        const int z = r % P.tnz; r /= P.tnz;
        const size_t addr = (size_t)((z + P.tz0) * (int)P.dimxy + (y + P.ty0) * P.nx + (x + P.tx0)) +
                            (size_t)(r + P.tg0) * P.nvox;
        field_add_large(P, addr, v);
    }
    // FP64 only here: per-thread FP32 partial sums reduced in double
    for (int k = 0; k < kNumEnergy; k++) {
        double v = (double)S.tally[k * B + tid];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(kFull, v, o);
        if (lane == 0 && v != 0.0) atomicAdd(P.energy + k, v);
    }
    const unsigned cnt[6] = {S.steps[tid], c_scat, c_dep, (lane == 0) ? S.wcount[2 * warp] : 0u,
                             (lane == 0) ? S.wcount[2 * warp + 1] : 0u, c_tile};
    const int cidx[6] = {kCntSteps, kCntScatter, kCntDeposit, kCntLaunch, kCntPhoton, kCntTileDeposit};
#pragma unroll
    for (int k = 0; k < 6; k++) {
        unsigned long long v = cnt[k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(kFull, v, o);
        if (lane == 0 && v) atomicAdd(P.counters + cidx[k], v);
    }
}
