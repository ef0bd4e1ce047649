// P2G with one thread per grid cell (included by mpm_kernels.cu).
//
// 64 threads (128 or 256 in small scenes of few blocks) take one 4x4x4-cell block of the sorted
// particle list:
//   1. the block's cell ranges come from the per-cell starts of the sort;
//   2. the threads of cell c walk its particles in sorted order, loading each one a particle ahead,
//      turn it into the affine contribution u + i*a0 + j*a1 + k*a2 (MLS / PB-MPM) and
//      accumulate the 27 stencil nodes in registers (the sums inside a block are deterministic);
//   3. a 27-phase flush adds the registers into a per-warp shared-memory 6x6x6 node tile: in one
//      phase the 32 lanes of a warp write 32 distinct nodes, so no atomics are needed;
//   4. the warp tiles are summed in a fixed order and each touched node gets one float4
//      vector atomic in the block-major accumulation grid.
// Particles whose stencil base lies outside the grid take a per-particle path with global vector
// atomics instead, and particles beyond the first kCellRun of a thread are added by vector atomics.
#pragma once

namespace crb200
{
    constexpr int kRec = 16;       // floats of a particle's P2G record
    // Records lie in tiles of 32 particles (2 KB): the first halves of the 32 records, then the second
    // halves.  A half is one 32-byte sector, so a gathered record costs two sectors as in one piece,
    // and a warp that writes 32 records touches 8 cache lines per store instead of 16.
    // Against whole 64-byte records: G2P 111 -> 106 us on a slab of 1.6M particles and 118 -> 114 us
    // over 64 scenes (1.3M); the cell accumulation reads either form in the same 71 us.
    constexpr unsigned kRecTile = 32, kRecHalf = 2 * kRecTile; // in float4
    __host__ __device__ __forceinline__ size_t recordAt(unsigned id)
    {
        return 4ull * (id & ~(kRecTile - 1u)) + 2u * (id & (kRecTile - 1u));
    }
    constexpr int kCellRun = 9;    // particles a cell thread accumulates; the rest of a cell's
                                   // particles go through per-particle vector atomics

    // Particles up to which a cell gets 4 threads, and 2 (see k_accumulate).
    constexpr unsigned kSplit4 = 30000, kSplit2 = 100000, kSplit4Batch = 12000, kSplit2Batch = 48000;

    // Per-particle scatter with global vector atomics (outliers and oversized blocks).
    // Mode 0 MLS, 1 PB (u/a already include the mass), 2 standard momentum, 3 standard force.
    template <int Mode>
    __device__ __forceinline__ void scatterGlobal(const StepParams &p, const Stencil &st, const float *rec,
                                                  unsigned cutMask, float4 *__restrict__ gridA, float4 *__restrict__ gridF)
    {
        const GridGeom &g = p.g;
        float w[3][3], dw[3][3];
        weights(st.fx, w);
        if (Mode == 3)
            weightGrads(st.fx, dw);
        const V3 u = v3(rec[0], rec[1], rec[2]);
        const float m = rec[3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j)
#pragma unroll
                for (int k = 0; k < 3; ++k)
                {
                    const int ni = st.b[0] + i, nj = st.b[1] + j, nk = st.b[2] + k;
                    if (!inGrid(g, ni, nj, nk) || ((cutMask >> (i * 9 + j * 3 + k)) & 1u))
                        continue;
                    const float wt = w[i][0] * w[j][1] * w[k][2];
                    const unsigned a = nodeAddr(g, ni, nj, nk);
                    if (Mode == 3)
                    {
                        const V3 gw = v3(dw[i][0] * w[j][1] * w[k][2], w[i][0] * dw[j][1] * w[k][2],
                                         w[i][0] * w[j][1] * dw[k][2]);
                        const float wm = wt * m;
                        const V3 f = v3(p.gravity.x * wm + rec[4] * gw.x + rec[7] * gw.y + rec[10] * gw.z,
                                        p.gravity.y * wm + rec[5] * gw.x + rec[8] * gw.y + rec[11] * gw.z,
                                        p.gravity.z * wm + rec[6] * gw.x + rec[9] * gw.y + rec[12] * gw.z);
                        atomicAdd(&gridF[a], make_float4(f.x, f.y, f.z, 0.f));
                    }
                    else
                    {
                        V3 val = u;
                        if (Mode <= 1)
                            val = u + v3(rec[4], rec[5], rec[6]) * (float)i + v3(rec[7], rec[8], rec[9]) * (float)j +
                                  v3(rec[10], rec[11], rec[12]) * (float)k;
                        atomicAdd(&gridA[a], make_float4(val.x * wt, val.y * wt, val.z * wt, m * wt));
                    }
                }
    }

    // Raw particle data a P2G thread needs (loaded one particle ahead of its use).
    struct RawParticle
    {
        float4 x4, v4, mp;
        float F[9], C[9];
        float v0;
        int mt;
    };

    template <int Mode>
    __device__ __forceinline__ void loadRaw(unsigned id, const float4 *__restrict__ xm, const float4 *__restrict__ vel,
                                            const float4 *__restrict__ matParams, const int *__restrict__ matType,
                                            const float *__restrict__ F, const float *__restrict__ Cm,
                                            const float *__restrict__ V0, unsigned stride, RawParticle &r)
    {
        r.x4 = xm[id];
        r.v4 = vel[id];
        r.mp = matParams[id];
        r.mt = matType[id];
#pragma unroll
        for (int k = 0; k < 9; ++k)
            r.F[k] = F[k * stride + id];
        if (Mode != 2)
        {
#pragma unroll
            for (int k = 0; k < 9; ++k)
                r.C[k] = Cm[k * stride + id];
        }
        r.v0 = (Mode == 1) ? 0.f : V0[id];
    }

    // Record of one particle for the cell accumulation:
    //   [0..2] u, [3] m, [4..12] a0 a1 a2 (MLS / PB) or -V0*tau column-major (standard force),
    //   [13..15] fx.
    // Returns 0 when the particle must not go through the cell path (non-finite position or a
    // stencil base outside [0, n-2]); such particles are scattered here with global atomics when
    // scatterOutliers is set.  PB-MPM without Svd: -1, and nothing done, when the particle's rotation
    // needs the SVD.
    template <int Mode, bool Svd = true>
    __device__ __forceinline__ int buildRecord(const StepParams &p, unsigned id, const RawParticle &raw,
                                                unsigned cutMask, bool scatterOutliers, float4 *__restrict__ gridA,
                                                float4 *__restrict__ gridF, unsigned *fp64Count, float rec[kRec])
    {
        const GridGeom &g = p.g;
        const Stencil st = stencilOf(g, v3(raw.x4));
        const float m = raw.x4.w;
#pragma unroll
        for (int e = 0; e < kRec; ++e)
            rec[e] = 0.f;
        if (!st.finite)
            return 0;
        const V3 v = v3(raw.v4);
        M3 Fp;
#pragma unroll
        for (int e = 0; e < 9; ++e)
            Fp.m[e] = raw.F[e];
        const float dx = g.dx;
        if (Mode == 0 || Mode == 1)
        {
            M3 A, Cp;
#pragma unroll
            for (int e = 0; e < 9; ++e)
                Cp.m[e] = raw.C[e];
            V3 base;
            if (Mode == 0)
            {
                const M3 s = kirchhoffStress(Fp, raw.mp.x, raw.mp.y, raw.mt);
                const float coef = -p.dt * 4.f * g.invDx * g.invDx * raw.v0;
#pragma unroll
                for (int e = 0; e < 9; ++e)
                    A.m[e] = s.m[e] * coef + Cp.m[e] * m;
                base = (v + v3(p.gravity) * p.dt) * m;
            }
            else
            {
                if (raw.mt == 1 || raw.mt == 0)
                {
                    // solveMaterialConstraints (constitutive_models.h:123-156)
                    M3 tF;
#pragma unroll
                    for (int e = 0; e < 9; ++e)
                        tF.m[e] = Cp.m[e] * p.dt + ((e % 4) == 0 ? 1.f : 0.f);
                    tF = matmul(tF, Fp);
                    M3 R;
                    if (Svd)
                        R = pbRotationTarget(tF, fp64Count);
                    else if (!pbRotationNear(tF, R))
                        return -1;
                    const float detF = det3(tF);
                    const float cd = fminf(fmaxf(fabsf(detF), 0.1f), 1000.0f);
                    const float qs = 1.0f / (copysignf(1.0f, detF) * sqrtf(cd));
                    M3 tgt;
#pragma unroll
                    for (int e = 0; e < 9; ++e)
                        tgt.m[e] = R.m[e] * raw.mp.y + (tF.m[e] * qs) * (1.0f - raw.mp.y);
                    const M3 TF = matmul(tgt, inverse3(Fp));
#pragma unroll
                    for (int e = 0; e < 9; ++e)
                        Cp.m[e] = Cp.m[e] + ((TF.m[e] - ((e % 4) == 0 ? 1.f : 0.f)) - Cp.m[e] * p.dt) * raw.mp.x;
                }
#pragma unroll
                for (int e = 0; e < 9; ++e)
                    A.m[e] = Cp.m[e] * m;
                base = v * m;
            }
            // u = base - A (fx dx); a_c = dx * A column c
            const V3 fd = v3(st.fx.x * dx, st.fx.y * dx, st.fx.z * dx);
            rec[0] = base.x - (A.m[0] * fd.x + A.m[3] * fd.y + A.m[6] * fd.z);
            rec[1] = base.y - (A.m[1] * fd.x + A.m[4] * fd.y + A.m[7] * fd.z);
            rec[2] = base.z - (A.m[2] * fd.x + A.m[5] * fd.y + A.m[8] * fd.z);
#pragma unroll
            for (int e = 0; e < 9; ++e)
                rec[4 + e] = A.m[e] * dx;
        }
        else
        {
            // standard MPM: momentum v m, force -V0 tau grad w + g w m (standard_mpm_algorithm.h:166-206)
            const M3 s = kirchhoffStress(Fp, raw.mp.x, raw.mp.y, raw.mt);
            const float nv0 = -raw.v0;
            rec[0] = v.x * m;
            rec[1] = v.y * m;
            rec[2] = v.z * m;
#pragma unroll
            for (int e = 0; e < 9; ++e)
                rec[4 + e] = s.m[e] * nv0;
        }
        rec[3] = m;
        rec[13] = st.fx.x;
        rec[14] = st.fx.y;
        rec[15] = st.fx.z;
        const bool inside = st.b[0] >= 0 && st.b[0] <= g.n.x - 2 && st.b[1] >= 0 && st.b[1] <= g.n.y - 2 &&
                            st.b[2] >= 0 && st.b[2] <= g.n.z - 2;
        if (!inside)
        {
            if (!scatterOutliers)
                return 0;
            if (Mode == 2)
            {
                scatterGlobal<2>(p, st, rec, 0u, gridA, gridF);
                scatterGlobal<3>(p, st, rec, 0u, gridA, gridF);
            }
            else
                scatterGlobal<Mode>(p, st, rec, cutMask, gridA, gridF);
            return 0;
        }
        return 1;
    }

    __device__ __forceinline__ void storeRecord(float4 *__restrict__ records, unsigned id, const float rec[kRec])
    {
        float4 *out = records + recordAt(id);
        out[0] = make_float4(rec[0], rec[1], rec[2], rec[3]);
        out[1] = make_float4(rec[4], rec[5], rec[6], rec[7]);
        out[kRecHalf] = make_float4(rec[8], rec[9], rec[10], rec[11]);
        out[kRecHalf + 1] = make_float4(rec[12], rec[13], rec[14], rec[15]);
    }

    // PB-MPM record of a particle whose rotation needs the SVD: out of line, so that its registers
    // do not limit the kernel around it.
    static __device__ __noinline__ void pbRecordSvd(const StepParams &p, unsigned id, RawParticle raw, unsigned msk,
                                                    float4 *__restrict__ gridA, unsigned *fp64Count,
                                                    float4 *__restrict__ records)
    {
        float rec[kRec];
        if (!buildRecord<1>(p, id, raw, msk, true, gridA, nullptr, fp64Count, rec))
        {
#pragma unroll
            for (int e = 0; e < kRec; ++e)
                rec[e] = 0.f;
        }
        storeRecord(records, id, rec);
    }

    // Adds one particle's 27 node contributions to the cell thread's registers.
    template <int Mode, bool Masked>
    __device__ __forceinline__ void accumulateCell(const StepParams &p, const float rec[kRec], unsigned msk, int pass,
                                                   float acc[27][4])
    {
        const V3 u = v3(rec[0], rec[1], rec[2]);
        const float m = rec[3];
        const V3 a0 = v3(rec[4], rec[5], rec[6]);
        const V3 a1 = v3(rec[7], rec[8], rec[9]);
        const V3 a2 = v3(rec[10], rec[11], rec[12]);
        const V3 fx = v3(rec[13], rec[14], rec[15]);
        float w[3][3], dw[3][3];
        weights(fx, w);
        if (Mode == 2 && pass == 1)
            weightGrads(fx, dw);
#pragma unroll
        for (int i = 0; i < 3; ++i)
        {
            const V3 ui = i == 0 ? u : fma3(a0, (float)i, u);
#pragma unroll
            for (int j = 0; j < 3; ++j)
            {
                const V3 uij = j == 0 ? ui : fma3(a1, (float)j, ui);
                const float wij = w[i][0] * w[j][1];
#pragma unroll
                for (int k = 0; k < 3; ++k)
                {
                    const int n = i * 9 + j * 3 + k;
                    if (Masked && ((msk >> n) & 1u))
                        continue;
                    const float wt = wij * w[k][2];
                    if (Mode == 2 && pass == 1)
                    {
                        const float wm = wt * m;
                        const float gx = dw[i][0] * w[j][1] * w[k][2], gy = w[i][0] * dw[j][1] * w[k][2],
                                    gz = wij * dw[k][2];
                        acc[n][0] += p.gravity.x * wm + a0.x * gx + a1.x * gy + a2.x * gz;
                        acc[n][1] += p.gravity.y * wm + a0.y * gx + a1.y * gy + a2.y * gz;
                        acc[n][2] += p.gravity.z * wm + a0.z * gx + a1.z * gy + a2.z * gz;
                    }
                    else if (Mode == 2)
                    {
                        acc[n][0] += u.x * wt;
                        acc[n][1] += u.y * wt;
                        acc[n][2] += u.z * wt;
                        acc[n][3] += m * wt;
                    }
                    else
                        fma4acc(acc[n], k == 0 ? uij : fma3(a2, (float)k, uij), m, wt);
                }
            }
        }
    }

    // (b) Every binned particle into its cell's slots, and its P2G record (indexed by particle id)
    //     unless the previous substep's G2P wrote it (carried; a scene with a slicer carries none,
    //     since its records follow the cut masks, which are evaluated here for MLS-MPM).  Outliers
    //     are scattered with global atomics and leave a zero record.  PB-MPM's relaxed C lives in the
    //     record only: G2P replaces C in the same iteration.
    //     Placing alone is a chain of three dependent accesses per particle: where nothing but that
    //     is left to do (carried, no slicer in any scene), a thread takes kPlacePer particles, so
    //     that as many chains are in flight, and the CTAs past the last particle exit: a substep of
    //     1.6M particles 218 -> 212 us.
    constexpr unsigned kPlacePer = 4, kPlaceThreads = 256;
    template <int Mode, bool Multi>
    __global__ void __launch_bounds__(kPlaceThreads, Mode == 1 ? 2 : 4) k_place(const __grid_constant__ StepParams p0, SceneTable sc,
                                                    bool carried, const unsigned *__restrict__ keys,
                                                    const unsigned *__restrict__ ranks, const unsigned *__restrict__ cellStart,
                                                    unsigned *__restrict__ sortedIds, unsigned capacity,
                                                    const float4 *__restrict__ xm,
                                                    const float4 *__restrict__ vel, const float4 *__restrict__ matParams,
                                                    const int *__restrict__ matType, const float *__restrict__ F,
                                                    const float *__restrict__ Cm, const float *__restrict__ V0, unsigned stride,
                                                    const ShapeRec *__restrict__ shapeTable, SdfPtrs sdf,
                                                    unsigned *__restrict__ cutMasks, float4 *__restrict__ records,
                                                    float4 *__restrict__ gridA, float4 *__restrict__ gridF, unsigned *fp64Count)
    {
        chainStart(p0.earlyNext);
        const unsigned n = Multi ? sc.numParticles : p0.numActive;
        const bool anyCut = Mode == 0 && (Multi || p0.numShapes > 0) && (*sc.anyFlags & SF_SLICER);
        const bool cutScene = !Multi && anyCut;
        const bool placeOnly = Mode == 0 && carried && !anyCut;
        const unsigned per = placeOnly ? kPlacePer : 1u;
        const unsigned i0 = blockIdx.x * kPlaceThreads * per + threadIdx.x;
        if (blockIdx.x * kPlaceThreads * per >= n)
            return;
        unsigned key[kPlacePer], slot[kPlacePer];
#pragma unroll
        for (unsigned e = 0; e < kPlacePer; ++e)
        {
            const unsigned i = i0 + kPlaceThreads * e;
            key[e] = e < per && i < n ? keys[i] : kInvalidKey;
            slot[e] = key[e] != kInvalidKey ? ranks[i] : 0u;
        }
#pragma unroll
        for (unsigned e = 0; e < kPlacePer; ++e)
            if (key[e] != kInvalidKey)
                slot[e] += cellStart[key[e]];
#pragma unroll
        for (unsigned e = 0; e < kPlacePer; ++e)
            if (key[e] != kInvalidKey && slot[e] < capacity) // always, unless the counts were inconsistent (flagged)
                sortedIds[slot[e]] = i0 + kPlaceThreads * e;
        if (placeOnly)
            return;
        __shared__ ShapeRec sh[Mode == 0 && !Multi ? kMaxShapes : 1];
        if (cutScene)
        {
            loadShapes(sh, shapeTable, p0.numShapes);
            __syncthreads();
        }
        const unsigned id = i0;
        // The masks are handed out (CrB200SolverCopyCutMasks): zero for a particle that takes no part, and
        // in a batch, whose masks are copied whole, for a scene without a slicer (once per call).
        const bool handsOut = Mode == 0 && (Multi ? p0.numShapes > 0 : cutScene);
        if (key[0] == kInvalidKey)
        {
            if (handsOut && id < n)
                cutMasks[id] = 0u;
            return;
        }
        const unsigned si = Multi ? sc.particleScene[id] : 0u; // sorted particles have a scene
        const StepParams &p = Multi ? sc.params[si] : p0;
        const bool slicers = Mode <= 1 && p.numShapes > 0 && (sc.flags[si] & SF_SLICER);
        if (Mode == 0 && carried && !slicers)
            return; // the previous G2P wrote this particle's record
        unsigned msk = 0u;
        if (slicers)
        {
            if (Mode == 0)
            {
                const V3 x = v3(xm[id]);
                msk = cutMaskOf(p.g, x, stencilOf(p.g, x), Multi ? shapeTable + p.shapeBegin : sh, p.numShapes, sdf);
                cutMasks[id] = msk;
            }
            else
                msk = cutMasks[id];
        }
        else if (Multi && handsOut)
            cutMasks[id] = 0u;
        RawParticle raw;
        loadRaw<Mode>(id, xm, vel, matParams, matType, F, Cm, V0, stride, raw);
        float rec[kRec];
        if (!buildRecord<Mode>(p, id, raw, msk, true, gridA, gridF, fp64Count, rec))
        {
#pragma unroll
            for (int e = 0; e < kRec; ++e)
                rec[e] = 0.f;
        }
        storeRecord(records, id, rec);
    }

    __device__ __forceinline__ void loadRecord(const float4 *__restrict__ records, unsigned j, float rec[kRec])
    {
        const float4 *r = records + recordAt(j);
        const float4 a = __ldg(r), b = __ldg(r + 1), c = __ldg(r + kRecHalf), d = __ldg(r + kRecHalf + 1);
        rec[0] = a.x; rec[1] = a.y; rec[2] = a.z; rec[3] = a.w;
        rec[4] = b.x; rec[5] = b.y; rec[6] = b.z; rec[7] = b.w;
        rec[8] = c.x; rec[9] = c.y; rec[10] = c.z; rec[11] = c.w;
        rec[12] = d.x; rec[13] = d.y; rec[14] = d.z; rec[15] = d.w;
    }

    // Groups of 64 threads in a CTA of the cell accumulation (see k_accumulate).
    template <int Split>
    constexpr int kGroups = Split == 4 ? 6 : Split;

    // Shared memory of a CTA of the cell accumulation, whose groups may each have a block of their own.
    template <bool Multi, int Split>
    struct AccumulateShared
    {
        static constexpr int kWarps = 2 * kGroups<Split>;
        // Node tile of each warp: momentum and mass of node (x, y, z) at x + kPitch (y + 6 z).  With a
        // pitch of 12 the 8 lanes of a 16-byte access (4 cells in x, 2 in y) cover all bank groups;
        // the widest CTAs, with 8 or 12 tiles, would pass 48 KB and take two-way conflicts.  One array of
        // float4 instead of four of floats: a quarter of the flush's instructions; a substep of
        // 1.6M particles 212 -> 209 us, of 85k 31.3 -> 31.1 us.
        static constexpr int kPitch = Split <= 2 ? 12 : kTileEdge, kTileSlots = kPitch * kTileEdge * kTileEdge;
        float4 tile[kWarps][kTileSlots];
        unsigned start[kGroups<Split>][65];
        unsigned ov[kGroups<Split>][65];
        unsigned warpTot[kGroups<Split>];
        StepParams p[Multi ? kGroups<Split> : 1]; // Multi: the current block's scene parameters
    };

    // The active blocks of a CTA, each worked on by a team of Step groups: Split groups, all on one block at a
    // time, or single groups with blocks of their own.
    template <int Mode, bool Multi, bool Det, int Split, int Step>
    __device__ __forceinline__ void accumulateBlocks(AccumulateShared<Multi, Split> &sh, const StepParams &p0,
                                                     const SceneTable &sc, unsigned nAct,
                                                     const unsigned *__restrict__ activeList,
                                                     const unsigned *__restrict__ blockEnd,
                                                     const unsigned *__restrict__ sortedIds,
                                                     const unsigned *__restrict__ cellStart,
                                                     const float4 *__restrict__ records,
                                                     const unsigned *__restrict__ cutMasks, float4 *__restrict__ gridA,
                                                     float4 *__restrict__ gridF, float4 *__restrict__ tiles,
                                                     float4 *__restrict__ tilesF)
    {
        constexpr bool kWhole = Step == Split; // one team; groups past it have nothing to do
        constexpr int kThreads = 64 * Step, kWarps = 2 * Step;
        constexpr unsigned kRun = (unsigned)(kCellRun * Step); // particles of a cell its threads take
        constexpr int kPitch = AccumulateShared<Multi, Split>::kPitch, kTileSlots = AccumulateShared<Multi, Split>::kTileSlots;
        if (kWhole && threadIdx.x >= (unsigned)kThreads)
            return;
        const unsigned team = kWhole ? 0u : threadIdx.x >> 6;
        const int tid = (int)(threadIdx.x - 64u * team), lane = tid & 31, warp = tid >> 5; // within the team
        const int cell = tid & 63; // the thread's cell; its particles are part, part + Step, ...
        const unsigned part = (unsigned)tid >> 6;
        unsigned *sStart = sh.start[team], *sOv = sh.ov[team];
        unsigned &sWarpTot = sh.warpTot[team];
        StepParams &sP = sh.p[Multi ? team : 0u];
        float4(*teamTile)[kTileSlots] = sh.tile + 2 * team;
        auto teamSync = [&]() {
            if constexpr (Split == 1)
                __syncthreads();
            else
                asm volatile("bar.sync %0, %1;" ::"r"(kWhole ? 0u : 1u + team), "n"(kThreads) : "memory");
        };
        // A record is loaded into registers while its predecessor is worked on, but for standard MPM with more
        // than one thread per cell: its second pass would spill (64k particles, 10 substeps 394 -> 384 us).
        constexpr bool kAhead = !(Mode == 2 && Split > 1);
        const int passes = Mode == 2 ? 2 : 1;
        const int cx = cell & 3, cy = (cell >> 2) & 3, cz = cell >> 4;
        for (unsigned ab = blockIdx.x + team * gridDim.x; ab < nAct; ab += gridDim.x * (kWhole ? 1u : (unsigned)kGroups<Split>))
        {
            const unsigned b = activeList[ab];
            const unsigned si = Multi ? (unsigned)sceneOfBlock(sc, b) : 0u;
            if (Multi)
            {
                // read at the use sites from shared memory rather than held in registers
                constexpr int words = (int)(sizeof(StepParams) / sizeof(unsigned));
                static_assert(words <= 64, "StepParams must fit one load per thread");
                if (tid < words)
                    reinterpret_cast<unsigned *>(&sP)[tid] = reinterpret_cast<const unsigned *>(&sc.params[si])[tid];
                teamSync();
            }
            const StepParams &p = Multi ? sP : p0;
            const GridGeom &g = p.g;
            const bool slicers = Mode <= 1 && p.numShapes > 0 && (sc.flags[si] & SF_SLICER);
            const unsigned lb = b - g.blockBase;
            const int bx = lb % g.nb.x, by = (lb / g.nb.x) % g.nb.y, bz = lb / (g.nb.x * g.nb.y);
            const unsigned start = cellStart[b * 64u], cnt = blockEnd[b] - start;
            // cell ranges of this block's sorted slots (cells are contiguous, in cell order)
            {
                unsigned oinc = 0;
                if (tid < 64)
                {
                    const unsigned excl = cellStart[b * 64u + tid] - start;
                    const unsigned v = (tid < 63 ? cellStart[b * 64u + tid + 1] - start : cnt) - excl;
                    sStart[tid] = excl;
                    if (tid == 63)
                        sStart[64] = cnt;
                    // overflow prefix: particles beyond the first kRun of each cell
                    oinc = v > kRun ? v - kRun : 0u;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1)
                    {
                        const unsigned y = __shfl_up_sync(0xffffffffu, oinc, o);
                        if (lane >= o)
                            oinc += y;
                    }
                }
                teamSync();
                if (tid == 31)
                    sWarpTot = oinc;
                teamSync();
                if (tid < 64)
                    sOv[tid + 1] = oinc + (warp ? sWarpTot : 0u);
                if (tid == 0)
                    sOv[0] = 0;
            }
            teamSync();
            const unsigned cs = sStart[cell] + part, ce = sStart[cell + 1];
            // Det: a cell thread takes all of its cell's particles, so nothing goes through atomics
            const unsigned runEnd = Det ? ce : min(ce, sStart[cell] + kRun);
            for (int pass = 0; pass < passes; ++pass)
            {
                float acc[27][4];
#pragma unroll
                for (int n = 0; n < 27; ++n)
                {
                    acc[n][0] = 0.f;
                    acc[n][1] = 0.f;
                    acc[n][2] = 0.f;
                    acc[n][3] = 0.f;
                }
                float nxt[kRec];
                unsigned nid = cs < runEnd ? sortedIds[start + cs] : 0u;
                if (kAhead && cs < runEnd)
                    loadRecord(records, nid, nxt);
                for (unsigned q = cs; q < runEnd; q += Step)
                {
                    float rec[kRec];
                    if (!kAhead)
                        loadRecord(records, nid, rec);
                    else
                    {
#pragma unroll
                        for (int e = 0; e < kRec; ++e)
                            rec[e] = nxt[e];
                    }
                    const unsigned id = nid;
                    if (q + Step < runEnd)
                    {
                        nid = sortedIds[start + q + Step];
                        if (kAhead)
                            loadRecord(records, nid, nxt);
                        else
                        {
                            const float4 *ahead = records + recordAt(nid);
                            asm volatile("prefetch.global.L1 [%0];" ::"l"(ahead));
                            asm volatile("prefetch.global.L1 [%0];" ::"l"(ahead + kRecHalf));
                        }
                    }
                    if (kAhead && q + 2 * Step < runEnd)
                    {
                        // the record after next into L1 (no registers held for it)
                        const float4 *ahead = records + recordAt(sortedIds[start + q + 2 * Step]);
                        asm volatile("prefetch.global.L1 [%0];" ::"l"(ahead));
                        asm volatile("prefetch.global.L1 [%0];" ::"l"(ahead + kRecHalf));
                    }
                    const unsigned msk = slicers ? cutMasks[id] : 0u;
                    if (msk)
                        accumulateCell<Mode, true>(p, rec, msk, pass, acc);
                    else
                        accumulateCell<Mode, false>(p, rec, 0u, pass, acc);
                }
                // phased flush of the registers into this warp's tile
                float4 *tile = teamTile[warp] + cx + kPitch * (cy + kTileEdge * cz);
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int j = 0; j < 3; ++j)
#pragma unroll
                        for (int k = 0; k < 3; ++k)
                        {
                            const int n = i * 9 + j * 3 + k;
                            float4 *t = tile + i + kPitch * (j + kTileEdge * k);
                            float4 v = *t;
                            v.x += acc[n][0];
                            v.y += acc[n][1];
                            v.z += acc[n][2];
                            v.w += acc[n][3];
                            *t = v;
                            __syncwarp();
                        }
                teamSync();
                // fixed-order sum of the warp tiles, one vector atomic per touched node
                for (int t = tid; t < kTileNodes; t += kThreads)
                {
                    const int tx = t % kTileEdge, tyz = t / kTileEdge;
                    const int e = tx + kPitch * tyz;
                    float4 v = teamTile[0][e];
                    teamTile[0][e] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int w = 1; w < kWarps; ++w)
                    {
                        const float4 o = teamTile[w][e];
                        teamTile[w][e] = make_float4(0.f, 0.f, 0.f, 0.f);
                        v = make_float4(v.x + o.x, v.y + o.y, v.z + o.z, v.w + o.w);
                    }
                    if (Det)
                    {
                        float4 *dst = (Mode == 2 && pass == 1) ? tilesF : tiles;
                        dst[(size_t)b * kTileNodes + t] = v;
                        continue;
                    }
                    const int i = 4 * bx + tx, j = 4 * by + tyz % kTileEdge, k = 4 * bz + tyz / kTileEdge;
                    if (!inGrid(g, i, j, k))
                        continue;
                    const unsigned a = nodeAddr(g, i, j, k);
                    if (Mode == 2 && pass == 1)
                    {
                        if (v.x != 0.f || v.y != 0.f || v.z != 0.f)
                            atomicAdd(&gridF[a], make_float4(v.x, v.y, v.z, 0.f));
                    }
                    else if (v.w != 0.f || v.x != 0.f || v.y != 0.f || v.z != 0.f)
                        atomicAdd(&gridA[a], v);
                }
                // particles beyond the first kRun of a cell: one per thread, vector atomics
                const unsigned total = Det ? 0u : sOv[64];
                for (unsigned kk = tid; kk < total; kk += kThreads)
                {
                    int lo = 0, hi = 63;
                    while (lo < hi)
                    {
                        const int mid = (lo + hi + 1) >> 1;
                        if (sOv[mid] <= kk)
                            lo = mid;
                        else
                            hi = mid - 1;
                    }
                    const unsigned slot = start + sStart[lo] + kRun + (kk - sOv[lo]);
                    float rec[kRec];
                    const unsigned sid = sortedIds[slot];
                    loadRecord(records, sid, rec);
                    if (rec[3] == 0.f && rec[0] == 0.f && rec[1] == 0.f && rec[2] == 0.f)
                        continue; // zero record (outlier already scattered, or massless)
                    Stencil st;
                    st.b[0] = 4 * bx + (lo & 3);
                    st.b[1] = 4 * by + ((lo >> 2) & 3);
                    st.b[2] = 4 * bz + (lo >> 4);
                    st.fx = v3(rec[13], rec[14], rec[15]);
                    st.finite = true;
                    const unsigned msk = slicers ? cutMasks[sid] : 0u;
                    if (Mode == 2 && pass == 0)
                        scatterGlobal<2>(p, st, rec, 0u, gridA, gridF);
                    else if (Mode == 2)
                        scatterGlobal<3>(p, st, rec, 0u, gridA, gridF);
                    else
                        scatterGlobal<Mode>(p, st, rec, msk, gridA, gridF);
                }
                teamSync();
            }
        }
    }

    // (c) Cell accumulation: groups of 64 threads, one thread per cell of an active block.
    //     Multi: each active block reads its scene's parameters.
    //     Det: nothing is added atomically.  A cell's threads accumulate all of its particles
    //     (no kCellRun cap) and the block's whole 6x6x6 tile is stored to tiles[block] (tilesF for
    //     the standard solver's force pass), from which the grid update sums each node's sources in
    //     a fixed order.
    //     Split: threads per cell, 1, 2 or 4 by the number of particles.  They take every Split-th particle
    //     of the cell, each with its own node sums and its warp with its own tile.  With one thread per cell
    //     a block is a serial walk of up to kCellRun particles, which is what the kernel costs while its
    //     blocks fit on the SMs at once; more threads shorten the walk but take the SM's registers from
    //     other blocks: 6, 3 and 1 blocks per SM are then worked on.  10 substeps with 1 / 2 / 4 threads
    //     per cell, us: 4096 particles 270 / 238 / 233, 22k 292 / 270 / 256, 64k 312 / 292 / 330, 111k
    //     338 / 335 / 396, 176k 437 / 460 / 521; standard MPM 64k 453 / 434 / 475; a PB-MPM step at 98k
    //     264 / 248 / 265, at 221k 361 / 377 / 431.  The lines (kSplit4 and so on) follow these at 8 particles
    //     per cell, with room for half as many; the blocks of a batch are less full (12k 315 / 297 /
    //     292, 40k 334 / 315 / 355, 70k 374 / 389 / 464).
    //     How many blocks that many particles lie in is known here only.  Where they are more than the CTAs
    //     (the resident ones: one round of them), the groups of a CTA take blocks of their own, one thread
    //     per cell, so that as many blocks are worked on as with 64-thread CTAs: 6 per SM with 2 threads
    //     per cell and, for the sake of this, 6 groups in the CTAs with 4.  10 substeps, us, all groups on
    //     one block -> on their own: 27k particles in 716 blocks 396 -> 273, PB-MPM 1585 -> 990, standard
    //     576 -> 372; 29k strewn over 6000 blocks 1714 -> 671, PB-MPM 8041 -> 2830, standard 2965 -> 1146;
    //     88k in 511 blocks 345 -> 334, PB-MPM 1344 -> 1332, standard 516 -> 518 (and 93k in 996, a last
    //     round of few blocks, 390 -> 368, 1558 -> 1484 and 586 -> 603).
    template <int Mode, bool Multi, bool Det, int Split>
    __global__ void __launch_bounds__(64 * kGroups<Split>, Split == 1 ? (Multi ? 5 : 6) : (Split == 2 ? 3 : 1)) k_accumulate(const __grid_constant__ StepParams p0, SceneTable sc, const SortHeader *__restrict__ hdr,
                                                       const unsigned *__restrict__ activeList,
                                                       const unsigned *__restrict__ blockEnd,
                                                       const unsigned *__restrict__ sortedIds,
                                                       const unsigned *__restrict__ cellStart,
                                                       const float4 *__restrict__ records,
                                                       const unsigned *__restrict__ cutMasks, float4 *__restrict__ gridA,
                                                       float4 *__restrict__ gridF, float4 *__restrict__ tiles,
                                                       float4 *__restrict__ tilesF)
    {
        chainStart(p0.earlyNext);
        __shared__ AccumulateShared<Multi, Split> sh;
        const unsigned nAct = hdr->numActiveBlocks;
        // each warp clears its own tile while the number of blocks is on its way
        for (int t = threadIdx.x & 31; t < sh.kTileSlots; t += 32)
            sh.tile[threadIdx.x >> 5][t] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncwarp();
        if (Split == 1 || nAct <= gridDim.x)
            accumulateBlocks<Mode, Multi, Det, Split, Split>(sh, p0, sc, nAct, activeList, blockEnd, sortedIds, cellStart, records,
                                                             cutMasks, gridA, gridF, tiles, tilesF);
        else
            accumulateBlocks<Mode, Multi, Det, Split, 1>(sh, p0, sc, nAct, activeList, blockEnd, sortedIds, cellStart, records,
                                                         cutMasks, gridA, gridF, tiles, tilesF);
    }
} // namespace crb200
