// Weight gradient on tcgen05, direct-sampling variant (included by dcn_tc.cu inside its anonymous namespace):
// each producer thread locates its own sampling points.  Fallback of dcn_tc_wgrad2.cuh for problems whose
// coordinate table does not fit in shared memory; also defines the work decomposition.
//
//   dW[o, k'] += sum over positions P of dy[o, P] * sample(k', P)          k' = tap * Cg + c
//
// GEMM view: M = output channels (128-row tiles, up to two per CTA), N = a block of up to 256 k' columns,
// K = output positions, 64 per pipeline stage.  One CTA owns one (group, o-block, k'-block) and a slice of
// the position range; partial sums are stored in a slice of the packed scratch of its own (see wg_slice_elems), and a
// fold job adds the slices in slice order into dW afterwards.
//   A operand: dy, bf16, pre-packed into swizzled [128 o][64 P] tiles  -> K-major, bulk-copied
//   B operand: sampled patch, [64 P rows][64 k' per 128-byte row] sub-tiles        -> MN-major, produced here
#pragma once

constexpr int kWgStages = 3;
constexpr int kWgNMax = 256;
// elements of one position split's slice of the packed dW scratch; `items` = G * MB * NB (the kernels' gridDim.x)
__host__ __device__ inline size_t wg_slice_elems(unsigned items) { return (size_t)items * 256 * kWgNMax; }
// Where a split keeps the sums of row (group, output channel) and columns kq..kq+3: [split][columns / 4][rows][4], so that
// the lanes of an epilogue warp (32 consecutive rows, four columns each) write 512 contiguous bytes.
struct WgDst {
    float4* base;
    size_t rows;
    __device__ __forceinline__ WgDst(float* dw, unsigned split, unsigned items, int NB, int row)
        : base(reinterpret_cast<float4*>(dw + split * wg_slice_elems(items)) + row), rows((size_t)(items / (unsigned)NB) * 256) {}
    __device__ __forceinline__ float4& at(int kq) const { return base[(size_t)(kq / 4) * rows]; }
};
constexpr int kWgThreads = 32 * (2 + kProducerWarps + kEpilogueWarps);

struct WgSmem {
    // per stage: A0 | A1 (16 KB each) | B (4 sub-tiles of 8 KB)
    static constexpr int kStageBytes = 2 * kTileBytes + 4 * 8192;
    static constexpr int kBarOffset = kWgStages * kStageBytes;
    static constexpr int kTotal = kBarOffset + (2 * kWgStages + 1) * 8 + 16;
};

template <int D, bool DEFORM>
__global__ void __launch_bounds__(kWgThreads, 1)
tc_wgrad_direct_kernel(const Geom g, const __nv_bfloat16* __restrict__ xcl, const float* __restrict__ off,
                const uint8_t* __restrict__ dpk, float* __restrict__ dw, const int MT, const int MB,
                const int NB, const int NW, const long long PC, const int chunks_per_split) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + WgSmem::kBarOffset);
    uint64_t* empty = full + kWgStages;
    uint64_t* acc_full = empty + kWgStages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;

    // work item of this CTA
    const int nb = blockIdx.x % NB;                     // k' block
    const int mb = (blockIdx.x / NB) % MB;              // o block (two 128-row tiles)
    const int j = blockIdx.x / NB / MB;                 // conv group
    const int mtb = (MT - mb * 2) >= 2 ? 2 : 1;
    const long long c_begin = (long long)blockIdx.y * chunks_per_split;
    long long c_end = c_begin + chunks_per_split;
    if (c_end > PC) c_end = PC;
    const int n_chunks = (int)(c_end - c_begin);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kWgStages; ++s) {
            mbar_init(&full[s], kProducerWarps + 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(acc_full, 1);
        fence_barrier_init();
    }
    pdl_wait();
    if (warp == 0) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t idesc = make_idesc(128, NW, 0, 1);   // A K-major, B MN-major

    if (warp == 0) {
        if (lane == 0) {
            bool ok = true;
            for (int it = 0; it < n_chunks && ok; ++it) {
                const uint32_t s = it % kWgStages;
                ok = mbar_wait(&full[s], (it / kWgStages) & 1);
                if (!ok) break;
                tc_fence_after();
                const uint32_t a_base = smem_u32(smem + s * WgSmem::kStageBytes);
                const uint32_t b_base = a_base + 2 * kTileBytes;
                for (int mt = 0; mt < mtb; ++mt) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint64_t ad = make_desc(a_base + mt * kTileBytes + k * 32, 16, 1024);
                        const uint64_t bd = make_desc(b_base + k * 2048, 8192, 1024);
                        umma_bf16(tmem_base + mt * 256, ad, bd, idesc, (it > 0 || k > 0) ? 1u : 0u);
                    }
                }
                umma_commit(&empty[s]);
            }
            if (ok) umma_commit(acc_full);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            bool ok = true;
            for (int it = 0; it < n_chunks && ok; ++it) {
                const uint32_t s = it % kWgStages;
                ok = mbar_wait(&empty[s], ((it / kWgStages) & 1) ^ 1);
                if (!ok) break;
                mbar_arrive_expect_tx(&full[s], (uint32_t)(mtb * kTileBytes));
                for (int mt = 0; mt < mtb; ++mt) {
                    const uint8_t* src = dpk + (((size_t)j * MT + mb * 2 + mt) * PC + (c_begin + it)) * kTileBytes;
                    bulk_g2s(smem + s * WgSmem::kStageBytes + mt * kTileBytes, src, kTileBytes, &full[s]);
                }
            }
        }
    } else if (warp < 2 + kProducerWarps) {
        const int ptid = threadIdx.x - 64;          // 0..255
        const int cj = ptid % 32;                   // k' chunk column (8 channels) inside the block
        const int row0 = ptid / 32;                 // rows row0 + 8*i
        const int kp = nb * kWgNMax + cj * 8;
        const bool kok = (cj * 8 < NW) && kp < g.kv * g.Cg;
        uint32_t tap = 0, cl = 0;
        g.d_Cg.divmod((uint32_t)(kok ? kp : 0), tap, cl);
        const int c = j * g.Cg + (int)cl;
        const int grp = (int)g.d_cpg.div((uint32_t)c);
        const uint32_t sub_off = (uint32_t)(cj / 8) * 8192u;
        bool ok = true;
        for (int it = 0; it < n_chunks && ok; ++it) {
            const uint32_t s = it % kWgStages;
            const long long Pc = (c_begin + it) * 64;
            uint4 v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                v[i] = make_uint4(0, 0, 0, 0);
                const long long P = Pc + row0 + 8 * i;
                if (kok && P < g.P) {
                    const OutPos op = decompose_pos(g, P);
                    v[i] = sample_chunk<D, DEFORM>(g, xcl, off, op, (int)tap, c, grp);
                }
            }
            ok = mbar_wait(&empty[s], ((it / kWgStages) & 1) ^ 1);
            if (!ok) break;
            if (cj * 8 < NW) {
                const uint32_t b_base = smem_u32(smem + s * WgSmem::kStageBytes + 2 * kTileBytes) + sub_off;
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    st_shared_v4(b_base + swz_offset(row0 + 8 * i, cj % 8), v[i].x, v[i].y, v[i].z, v[i].w);
            }
            fence_proxy_async_smem();
            mbar_arrive_warp(&full[s]);
        }
    } else {
        const int q = warp & 3;
        if (n_chunks > 0 && mbar_wait(acc_full, 0)) {
            tc_fence_after();
            for (int mt = 0; mt < mtb; ++mt) {
                const int ol = (mb * 2 + mt) * 128 + q * 32 + lane;
                const bool o_ok = ol < g.Og;
                // partial sums of this position split: plain stores into its slice of the packed scratch (added
                // up in split order by the dW fold)
                const WgDst dst(dw, blockIdx.y, gridDim.x, NB, j * MB * 256 + ol);
                for (int cc = 0; cc < NW / 32; ++cc) {
                    uint32_t v[32];
                    tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + mt * 256 + cc * 32, v);
                    tmem_ld_wait();
                    if (!o_ok) continue;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int kq = nb * kWgNMax + cc * 32 + 4 * i;
                        if (kq < g.kv * g.Cg)
                            dst.at(kq) =
                                make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]),
                                            __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3]));
                    }
                }
            }
        }
    }

    pdl_trigger();              // (late: a waiting block of the next kernel would take shared memory from this one's L1)
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

struct WgDims {
    int MT, MB, NB, NW;
    long long PC;
    int splits, cps;
};

inline WgDims wg_dims(const Geom& g) {
    WgDims d;
    d.MT = (g.Og + 127) / 128;
    d.MB = (d.MT + 1) / 2;
    const int kq = g.kv * g.Cg;
    d.NB = (kq + kWgNMax - 1) / kWgNMax;
    d.NW = kq >= kWgNMax ? kWgNMax : ((kq + 63) / 64) * 64;
    d.PC = 2 * ((g.P + 127) / 128);     // 64-position chunks, even count (shared tile layout with dgrad)
    const long long items = (long long)g.G * d.MB * d.NB;
    // position slices: CTAs in up to three waves, weighed in chunks of 64 positions, a CTA costing five beside its own
    // (set-up and epilogue; 2 us a chunk)
    const int S = sm_count();
    long long splits = 1, best = 0;
    for (long long k = 1; k <= d.PC && k <= 65535 && (k == 1 || items * k <= 3ll * S); ++k) {
        const long long c = (items * k + S - 1) / S * ((d.PC + k - 1) / k + 5);
        if (k == 1 || c < best) { best = c; splits = k; }
    }
    d.cps = (int)((d.PC + splits - 1) / splits);
    d.splits = (int)((d.PC + d.cps - 1) / d.cps);
    return d;
}

inline size_t dwpk_bytes(const Geom& g) {
    const WgDims d = wg_dims(g);
    return (size_t)d.splits * wg_slice_elems(g.G * d.MB * d.NB) * sizeof(float);
}

// the fold of the position splits' sums into dW (add: accumulate)
inline void add_dw_fold(Passes& p, const Geom& g, const float* dwpk, float* dw, bool add) {
    const WgDims d = wg_dims(g);
    p.fold_dw(g, dwpk, dw, d.MB * 256, d.splits, wg_slice_elems(g.G * d.MB * d.NB), add);
}

template <int D, bool DEFORM>
int launch_tc_wgrad_direct(const Geom& g, const __nv_bfloat16* xcl, const float* off, const uint8_t* dpk, float* dw,
                    cudaStream_t st) {
    const WgDims d = wg_dims(g);
    const int smem = WgSmem::kTotal + 1024;
    auto kern = tc_wgrad_direct_kernel<D, DEFORM>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -5;
    dim3 grid((unsigned)(g.G * d.MB * d.NB), (unsigned)d.splits);
    return launch_dependent(kern, grid, dim3(kWgThreads), smem, st, g, xcl, off, dpk, dw, d.MT, d.MB, d.NB, d.NW, d.PC,
                            d.cps) == cudaSuccess ? 0 : -5;
}
