// Forward implicit GEMM on tcgen05 (included by dcn_tc.cu inside its anonymous namespace).
//
//   y[o, P] = sum over k' of W[o, k'] * sample(k', P)  (+ bias)            k' = tap * Cg + c
//
// Persistent CTAs, one per SM; 6 + GW warps:
//   warp 0       MMA issue (one elected lane) and tensor-memory allocation
//   warp 1       weight-tile loader (bulk async copies, one elected lane)
//   warps 2-5    coordinate warps (dcn_tc_sampler.cuh).  Warp k fills the whole table of every 4th pipeline stage
//                (k, k+4, ...): the chain offsets -> coordinates -> corner table of one stage is long and serial,
//                so four stages are in production at once.  The same warps drain finished accumulators
//                (tensor memory -> registers -> (+bias) -> y) whenever they have no table to fill, so the
//                epilogue costs no warps of its own.
//   warps 6..    GW gather warps: build the sampled, interpolated patch tile straight into the swizzled B
//                operand, all of them on the same stage (splitting them into groups that take alternate
//                stages measured slower).
// Tile = (conv group, block of up to 256 output channels, 128 output positions).  The sampled operand of a
// K chunk is shared by both 128-row halves of the output-channel block.
#pragma once

constexpr int kMaxStages = 4;
constexpr int kFwdCoordWarps = 4;               // forward: coordinate + epilogue warps, one per tensor-memory lane quarter
constexpr int fwd_threads(int gw) { return 32 * (2 + kFwdCoordWarps + gw); }
constexpr int kFwdStageBytes = 3 * kTileBytes;      // A0 | A1 | B
constexpr int kSmemLimit = 232448;                   // 227 KB opt-in maximum per CTA

constexpr int kFwdMaxTabs = 6;
constexpr int kFwdOutBytes = kFwdCoordWarps * 32 * 33 * (int)sizeof(float);
constexpr int kFwdOffRing = 2 * kFwdCoordWarps;   // two private offset staging buffers per coordinate warp

struct FwdCtl {            // lives behind the stages, the tables and the offset staging ring
    uint64_t full[kMaxStages], empty[kMaxStages], acc_full[2], acc_empty[2], tab_full[kFwdMaxTabs], tab_empty[kFwdMaxTabs];
    uint32_t tmem_base;
    int slot_of_chunk[kFwdMaxTabs][8];
};

// How the work items of the persistent CTAs map to (tile, K range).  Items [0, T0) split every tile KS0 ways
// (KS0 = 1: whole tiles); items from T0 on split the tiles from tile1 on KS1 ways.  The second region is the
// tail of a grid that does not divide evenly: the tiles left over after the last full wave are split along K so
// that the last wave is a fraction of a tile long instead of a whole one.
// The items of split tiles store their sums in a slice of scratch each (item order); a fold behind the kernel adds
// the slices of a tile in K order and stores y (fold_y, dcn_tc_passes.cuh).
struct FwdSplit {
    long long T0, tile1, n_items;
    int KS0, cpk0, KS1, cpk1;
    int acc;            // y already holds a partial result, which the tiles are added to (plain convolution only)
};
struct FwdItem {
    long long tt;       // tile index ((j * MB + mb) * PT + pt)
    long long slice;    // of a split tile: where its sums go; else -1
    int kc0, kc1;       // its K chunks [kc0, kc1)
};
__device__ __forceinline__ FwdItem fwd_item(const FwdSplit& sp, long long t, int KC) {
    const bool tail = t >= sp.T0;
    const long long r = tail ? t - sp.T0 : t;
    const int KS = tail ? sp.KS1 : sp.KS0, cpk = tail ? sp.cpk1 : sp.cpk0;
    FwdItem it;
    it.tt = (tail ? sp.tile1 : 0) + r / KS;
    it.slice = KS > 1 ? r : -1;
    it.kc0 = (int)(r % KS) * cpk;
    it.kc1 = (it.kc0 + cpk < KC) ? it.kc0 + cpk : KC;
    return it;
}

// TURN: see FwdPlan::turn (a kernel of its own: with both epilogues in one the 3-D kernel spills, 1000 -> 1095 us)
template <int D, bool DEFORM, int GW, bool TURN>
__global__ void __launch_bounds__(fwd_threads(GW), 1)
tc_forward_kernel(const Geom g, const __nv_bfloat16* __restrict__ xcl, const float* __restrict__ off,
                  const uint8_t* __restrict__ wpk, const float* __restrict__ bias, float* __restrict__ y,
                  const int KC, const int MT, const int MB, const long long PT, const int n_stages,
                  const int max_slots, const int n_tabs, const FwdSplit sp, float* __restrict__ slices) {
    // Work items: see FwdSplit.  With few position tiles and a long K every tile is split (small batches, late
    // layers of a network); otherwise only the tiles of the last, partial wave are.
    using Entry = TabEntry<D, DEFORM>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    Entry* tab = reinterpret_cast<Entry*>(smem + n_stages * kFwdStageBytes);          // [n_tabs][max_slots][128]
    float* ostage = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(tab) +
                                             (size_t)n_tabs * max_slots * 128 * sizeof(Entry));   // [kFwdOffRing][max_slots][D][128]
    FwdCtl* ctl = reinterpret_cast<FwdCtl*>(ostage + (size_t)kFwdOffRing * max_slots * D * 128);
    float* obuf = reinterpret_cast<float*>(ctl + 1);                // turn: [kFwdCoordWarps][32][33], see the epilogue

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kMaxStages; ++s) {
            mbar_init(&ctl->full[s], GW + 1);            // one arrival per gather warp + the loader
            mbar_init(&ctl->empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&ctl->acc_full[b], 1);
            mbar_init(&ctl->acc_empty[b], kFwdCoordWarps);
        }
        for (int b = 0; b < kFwdMaxTabs; ++b) {
            mbar_init(&ctl->tab_full[b], 1);             // the coordinate warp that filled it
            mbar_init(&ctl->tab_empty[b], GW);           // the gather warps that read it
        }
        fence_barrier_init();
    }
    pdl_wait();
    if (warp == 0) {
        tmem_alloc(&ctl->tmem_base, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = ctl->tmem_base;

    const long long n_tiles = sp.n_items;
    constexpr uint32_t kIdesc = make_idesc(128, kTileN, 0, 0);

    if (warp == 0) {
        // ------------------------------------------------ MMA issue
        if (lane == 0) {
            uint32_t tl = 0;
            Ring rs;
            bool ok = true;
            for (long long t = blockIdx.x; t < n_tiles && ok; t += gridDim.x, ++tl) {
                const FwdItem wi = fwd_item(sp, t, KC);
                const long long tt = wi.tt;
                const int mb = (int)((tt / PT) % MB);
                const int mtb = (MT - mb * 2) >= 2 ? 2 : 1;
                const int kc0 = wi.kc0, kc1 = wi.kc1;
                const uint32_t b = tl & 1;
                ok = mbar_wait(&ctl->acc_empty[b], ((tl >> 1) & 1) ^ 1);
                tc_fence_after();
                for (int kc = kc0; kc < kc1 && ok; ++kc, rs.next(n_stages)) {
                    const uint32_t s = rs.i;
                    ok = mbar_wait(&ctl->full[s], rs.ph);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t a_base = smem_u32(smem + s * kFwdStageBytes);
                    const uint32_t b_base = a_base + 2 * kTileBytes;
                    // one descriptor per operand and stage; the K step and the second M tile only move the
                    // start-address field (units of 16 bytes), which cannot carry out of its 14 bits
                    const uint64_t ad0 = make_desc(a_base, 16, 1024);
                    const uint64_t bd0 = make_desc(b_base, 16, 1024);
                    for (int mt = 0; mt < mtb; ++mt) {
#pragma unroll
                        for (int k = 0; k < kTileK / 16; ++k) {
                            umma_bf16(tmem_base + b * 256 + mt * 128, ad0 + (uint64_t)((mt * kTileBytes + k * 32) >> 4),
                                      bd0 + (uint64_t)((k * 32) >> 4), kIdesc, (kc > kc0 || k > 0) ? 1u : 0u);
                        }
                    }
                    umma_commit(&ctl->empty[s]);
                }
                if (ok) umma_commit(&ctl->acc_full[b]);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------ weight loader
        if (lane == 0) {
            Ring rs;
            bool ok = true;
            for (long long t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
                const FwdItem wi = fwd_item(sp, t, KC);
                const long long tt = wi.tt;
                const int mb = (int)((tt / PT) % MB);
                const int j = (int)(tt / PT / MB);
                const int mtb = (MT - mb * 2) >= 2 ? 2 : 1;
                const int kc0 = wi.kc0, kc1 = wi.kc1;
                for (int kc = kc0; kc < kc1 && ok; ++kc, rs.next(n_stages)) {
                    const uint32_t s = rs.i;
                    ok = mbar_wait(&ctl->empty[s], rs.ph ^ 1u);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&ctl->full[s], (uint32_t)(mtb * kTileBytes));
                    for (int mt = 0; mt < mtb; ++mt) {
                        const uint8_t* src = wpk + ((size_t)(j * MT + mb * 2 + mt) * KC + kc) * kTileBytes;
                        bulk_g2s(smem + s * kFwdStageBytes + mt * kTileBytes, src, kTileBytes, &ctl->full[s]);
                    }
                }
            }
        }
    } else if (warp < 2 + kFwdCoordWarps) {
        // ------------------------------------------------ coordinate + epilogue warps
        const int cw = warp - 2;                    // takes stages cw, cw + 4, ... of this CTA's stage sequence
        const int q = warp & 3;                     // tensor-memory lane quarter this warp may access
        constexpr int CR = 4;                       // table rows per thread: lane + 32 * i
        struct Cur {
            long long t, pt;
            int kc, kc_end, j;
            uint32_t tl;            // how many tiles of this CTA came before t
        };
        auto init_tile = [&](Cur& c) {
            const FwdItem wi = fwd_item(sp, c.t, KC);
            c.pt = wi.tt % PT;
            c.j = (int)(wi.tt / PT / MB);
            c.kc = wi.kc0;
            c.kc_end = wi.kc1;
        };
        auto skip = [&](Cur& c, int n) {            // n stages further
            for (int i = 0; i < n && c.t < n_tiles; ++i) {
                if (++c.kc == c.kc_end) {
                    c.t += gridDim.x;
                    ++c.tl;
                    if (c.t < n_tiles) init_tile(c);
                }
            }
        };
        auto stage_slots = [&](const Cur& c) {
            int tap_, c_;
            const int key = chunk_key(g, c.j, c.kc * kTileK + (lane & 7) * 8, tap_, c_);
            return make_slots(key, lane, 8);
        };
        // Offsets of a stage are fetched with 4-byte cp.async into one of this warp's two staging buffers while
        // the warp's previous stage is being filled, so their latency is off the critical path.
        float* my_ost = ostage + (size_t)cw * 2 * max_slots * D * 128;
        auto prefetch = [&](const Cur& c, uint32_t buf) {
            if (DEFORM && c.t < n_tiles) {
                const SlotInfo si = stage_slots(c);
                float* dst = my_ost + (size_t)buf * max_slots * D * 128;
                for (int sl = 0; sl < si.nslots; ++sl) {
                    const int key = slot_key(si, sl);
                    if (key < 0) continue;
                    uint32_t grp, tap;
                    g.d_kv.divmod((uint32_t)key, grp, tap);
#pragma unroll
                    for (int i = 0; i < CR; ++i) {
                        const long long P = c.pt * kTileN + lane + 32 * i;
                        if (P >= g.P) continue;
                        const OutPos op = decompose_pos(g, P);
                        const float* src = offset_ptr<float, D>(g, offset_block<float, D>(g, off, op.n), (int)grp, (int)tap, op);
#pragma unroll
                        for (int a = 0; a < D; ++a)
                            cp_async4(dst + (size_t)(sl * D + a) * 128 + lane + 32 * i, src + (size_t)a * g.ov);
                    }
                }
            }
            cp_async_commit();
        };
        Cur cur;
        cur.t = blockIdx.x; cur.pt = 0; cur.kc = 0; cur.kc_end = 0; cur.j = 0; cur.tl = 0;
        if (cur.t < n_tiles) init_tile(cur);
        skip(cur, cw);
        Ring rt;
        for (int i = 0; i < cw; ++i) rt.next(n_tabs);
        prefetch(cur, 0);
        {
            Cur pre = cur;
            skip(pre, kFwdCoordWarps);
            prefetch(pre, 1);
        }
        uint32_t it = 0;                // stages this warp has filled
        long long et = blockIdx.x;      // next tile whose accumulator this warp drains
        uint32_t etl = 0;               // ... and how many tiles of this CTA came before it
        bool waiting = false;
        long long t0 = 0;
        while (true) {
            const bool more = cur.t < n_tiles;
            if (!more && et >= n_tiles) break;
            const bool tab_free = more && mbar_try_wait(&ctl->tab_empty[rt.i], rt.ph ^ 1u);
            // Drain an accumulator when there is no table to fill (the ring is full, or the tables are done) or
            // when the tables of the tile that needs the accumulator's buffer are about to be filled.
            if (et < n_tiles && (!tab_free || cur.tl >= etl + 2) &&
                mbar_try_wait(&ctl->acc_full[etl & 1], (etl >> 1) & 1)) {
                waiting = false;
                tc_fence_after();
                const uint32_t b = etl & 1;
                const FwdItem wi = fwd_item(sp, et, KC);
                const bool plain = DEFORM || sp.acc == 0;
                const long long tt = wi.tt;
                const long long pt = tt % PT;
                const int mb = (int)((tt / PT) % MB);
                const int j = (int)(tt / PT / MB);
                const int mtb = (MT - mb * 2) >= 2 ? 2 : 1;
                if (wi.slice >= 0) {
                    float* s = slices + (size_t)wi.slice * ((MT >= 2 ? 2 : 1) * kSliceHalf) + q * (kSliceHalf / 4) + lane * 4;
#pragma unroll 1
                    for (int c = 0; c < mtb * (kTileN / 16); ++c) {
                        const int mt = c / (kTileN / 16), cc = c % (kTileN / 16);
                        uint32_t v[16];
                        tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + b * 256 + mt * 128 + cc * 16, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            *reinterpret_cast<uint4*>(s + (size_t)mt * kSliceHalf + cc * kSliceGroup + i * 128) =
                                make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                    }
                } else
                for (int mt = 0; mt < mtb; ++mt) {
                    const int ol = (mb * 2 + mt) * 128 + q * 32 + lane;      // output channel within the group
                    const bool o_ok = ol < g.Og;
                    const int o = j * g.Og + ol;
                    const float bv = (bias != nullptr && o_ok) ? gload(bias + o) : 0.f;
                    if constexpr (TURN) {
                        // Channel-first y whose rows are not 16-byte aligned: 32 x 32 pieces are turned in shared memory
                        // and leave as 128-byte runs along the positions.  (A lane storing its own row of an odd size
                        // value by value touches 32 lines per instruction: 2 x 128 channels at 101x151, 67 us against
                        // 57 us.  Aligned rows stay with the 16-byte stores below, which are faster still.)
                        float* ob = obuf + cw * 32 * 33;
#pragma unroll 1
                        for (int cc = 0; cc < kTileN / 32; ++cc) {
                            const long long P = pt * kTileN + cc * 32 + lane;
                            if (pt * kTileN + cc * 32 >= g.P) break;
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                uint32_t v[16];
                                tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + b * 256 + mt * 128 + cc * 32 + h * 16, v);
                                tmem_ld_wait();
#pragma unroll
                                for (int i = 0; i < 16; ++i) ob[lane * 33 + h * 16 + i] = __uint_as_float(v[i]) + bv;
                            }
                            __syncwarp();
                            uint32_t n, opos;
                            g.d_ov.divmod((uint32_t)(P < g.P ? P : 0), n, opos);
                            const int o0 = (mb * 2 + mt) * 128 + q * 32;
                            float* d1 = y + ((size_t)n * g.O + j * g.Og + o0) * g.ov + opos;
                            const int rows = g.Og - o0 < 32 ? g.Og - o0 : 32;
                            if (P < g.P) {
#pragma unroll 4
                                for (int r = 0; r < rows; ++r, d1 += g.ov) {
                                    const float val = ob[r * 33 + lane];
                                    if (plain) *d1 = val;
                                    else atomicAdd(d1, val);
                                }
                            }
                            __syncwarp();
                        }
                    } else {
#pragma unroll 1
                    for (int cc = 0; cc < kTileN / 16; ++cc) {
                        uint32_t v[16];
                        tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + b * 256 + mt * 128 + cc * 16, v);
                        tmem_ld_wait();
                        const long long P0 = pt * kTileN + cc * 16;
                        if (!o_ok || P0 >= g.P) continue;
                        if (g.cl) {
                            // channels-last y: the 32 lanes of the warp hold 32 consecutive channels of a position
#pragma unroll
                            for (int i = 0; i < 16; ++i) {
                                if (P0 + i < g.P) {
                                    float* d1 = y + (size_t)(P0 + i) * g.O + o;
                                    if (plain) *d1 = __uint_as_float(v[i]) + bv;
                                    else atomicAdd(d1, __uint_as_float(v[i]) + bv);
                                }
                            }
                            continue;
                        }
                        uint32_t n0, opos0;
                        g.d_ov.divmod((uint32_t)P0, n0, opos0);
                        float* dst = y + ((size_t)n0 * g.O + o) * g.ov + opos0;
                        const bool fast = (opos0 + 16 <= (uint32_t)g.ov) && ((reinterpret_cast<uintptr_t>(dst) & 15) == 0);
                        if (fast) {
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const float4 val = make_float4(__uint_as_float(v[4 * i]) + bv, __uint_as_float(v[4 * i + 1]) + bv,
                                                               __uint_as_float(v[4 * i + 2]) + bv, __uint_as_float(v[4 * i + 3]) + bv);
                                if (plain) *reinterpret_cast<float4*>(dst + 4 * i) = val;
                                else atomicAdd(reinterpret_cast<float4*>(dst + 4 * i), val);
                            }
                        } else {
#pragma unroll
                            for (int i = 0; i < 16; ++i) {
                                const long long P = P0 + i;
                                if (P < g.P) {
                                    uint32_t n, opos;
                                    g.d_ov.divmod((uint32_t)P, n, opos);
                                    float* d1 = y + ((size_t)n * g.O + o) * g.ov + opos;
                                    if (plain) *d1 = __uint_as_float(v[i]) + bv;
                                    else atomicAdd(d1, __uint_as_float(v[i]) + bv);
                                }
                            }
                        }
                    }
                    }
                }
                tc_fence_before();
                mbar_arrive_warp(&ctl->acc_empty[b]);
                et += gridDim.x;
                ++etl;
                continue;
            }
            if (tab_free) {
                waiting = false;
                cp_async_wait<1>();             // this stage's offsets have landed; the next stage's may be in flight
                const uint32_t tb = rt.i;
                const SlotInfo si = stage_slots(cur);
                if (lane < 8) ctl->slot_of_chunk[tb][lane] = si.my_slot;
                const float* src = my_ost + (size_t)(it & 1u) * max_slots * D * 128;
                for (int sl = 0; sl < si.nslots; ++sl) {
                    const int key = slot_key(si, sl);
#pragma unroll
                    for (int i = 0; i < CR; ++i) {
                        const long long P = cur.pt * kTileN + lane + 32 * i;
                        const bool pok = P < g.P;
                        const OutPos op = decompose_pos(g, pok ? P : 0);
                        float offv[D];
#pragma unroll
                        for (int a = 0; a < D; ++a)
                            offv[a] = (DEFORM && key >= 0 && pok) ? src[(size_t)(sl * D + a) * 128 + lane + 32 * i] : 0.f;
                        fill_entry_from<D, DEFORM>(g, offv, op, pok, key, tab + ((size_t)tb * max_slots + sl) * 128 + lane + 32 * i);
                    }
                }
                mbar_arrive_warp(&ctl->tab_full[tb]);
                skip(cur, kFwdCoordWarps);
                for (int i = 0; i < kFwdCoordWarps; ++i) rt.next(n_tabs);
                {
                    Cur pre = cur;              // the stage after the next one goes into the buffer just read
                    skip(pre, kFwdCoordWarps);
                    prefetch(pre, it & 1u);
                }
                ++it;
                continue;
            }
            // nothing to do yet: bounded wait for either event
            __nanosleep(200);
            if (!waiting) {
                waiting = true;
                t0 = clock64();
            } else if (clock64() - t0 > kWaitCycles) {
                atomicOr(&g_tc_status, 1u);
                break;
            }
        }
        cp_async_wait<0>();
    } else {
        // ------------------------------------------------ gather warps
        // Within a thread a stage is produced in passes of RPP rows; where the registers allow it the loads
        // of the next pass are in flight while the current one is interpolated and stored.
        const int gtid = threadIdx.x - 32 * (2 + kFwdCoordWarps);   // 0..GW*32-1
        const int chunk = gtid % 8;                 // 16-byte chunk of the 128-byte row
        const int row0 = gtid / 8;                  // rows row0 + RS*i, i = 0..RT-1
        constexpr int NQ = DEFORM ? (1 << D) : 1;
        constexpr int RT = 128 * 8 / (GW * 32);     // rows per thread and stage
        constexpr int RS = GW * 4;                  // row stride between a thread's rows
        constexpr int RPP = (RT >= 2 && !(D == 3 && DEFORM && GW > 8)) ? 2 : 1;   // rows per pass (16 or 8 loads)
        constexpr int PPS = RT / RPP;               // passes per stage
        // 2-D: two passes in flight (16 loads); 3-D: one pass already has 16 loads in flight, and two would
        // not fit the register file.
        constexpr bool kOverlap = (D == 2 || !DEFORM) && PPS >= 2 && GW <= 10;
        struct Pass {
            uint4 q[RPP][NQ];
            float w[RPP][NQ];
            uint32_t s, ph;     // operand stage of this pass and the phase of its barriers
            int h;
        };
        // issue cursor: stage sequence (tile, K chunk) of this CTA
        long long ct = blockIdx.x, cpt = 0;
        int ckc = 0, ckc_end = 0, ch = 0, cj = 0, cc = 0, csl = 0;
        Ring rtab, rstg;            // table buffer and operand stage of the issue cursor
        bool failed = false;
        const uint32_t tab_s = smem_u32(tab);
        const uint32_t pix_bytes = (uint32_t)g.C * 2u;
        const __nv_bfloat16* xbase[RT];         // channels-last base of the sample of each of this thread's rows
        auto init_tile = [&]() {
            const FwdItem wi = fwd_item(sp, ct, KC);
            cpt = wi.tt % PT;
            cj = (int)(wi.tt / PT / MB);
            ckc = wi.kc0;
            ckc_end = wi.kc1;
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                const long long P = cpt * kTileN + row0 + RS * i;
                uint32_t n = 0;
                if (P < g.P) n = g.d_ov.div((uint32_t)P);
                xbase[i] = xcl + (uint64_t)(n * (uint32_t)g.iv) * (uint32_t)g.C;
            }
        };
        auto next_stage = [&]() {
            rtab.next(n_tabs);
            rstg.next(n_stages);
            if (++ckc == ckc_end) {
                ct += gridDim.x;
                if (ct < n_tiles) init_tile();
            }
        };
        if (ct < n_tiles) init_tile();
        auto issue = [&](Pass& p) -> bool {
            if (ct >= n_tiles || failed) return false;
            const uint32_t tb = rtab.i;
            if (ch == 0) {
                const bool okw = mbar_wait(&ctl->tab_full[tb], rtab.ph); if (!okw) { failed = true; return false; }
                csl = ctl->slot_of_chunk[tb][chunk];
                const int kp = ckc * kTileK + chunk * 8;
                uint32_t tap, cl;
                g.d_Cg.divmod((uint32_t)(kp < g.kv * g.Cg ? kp : 0), tap, cl);
                cc = cj * g.Cg + (int)cl;
            }
            const uint32_t trow_s = tab_s + ((tb * (uint32_t)max_slots + (uint32_t)csl) * 128u) * (uint32_t)sizeof(Entry);
#pragma unroll
            for (int hh = 0; hh < PPS; ++hh) {
                if (hh == ch) {
#pragma unroll
                    for (int r = 0; r < RPP; ++r) {
                        const int i = hh * RPP + r;
                        gather_issue_s<D, DEFORM>(trow_s + (uint32_t)(row0 + RS * i) * (uint32_t)sizeof(Entry),
                                                  xbase[i] + cc, pix_bytes, p.q[r], p.w[r]);
                    }
                }
            }
            p.s = rstg.i;
            p.ph = rstg.ph;
            p.h = ch;
            if (ch == PPS - 1) mbar_arrive_warp(&ctl->tab_empty[tb]);   // this warp is done with the stage's table
            if (++ch == PPS) {
                ch = 0;
                next_stage();
            }
            return true;
        };
        auto finish = [&](Pass& p) -> bool {
            const uint32_t s = p.s;
            if (p.h == 0) {
                const bool okw = mbar_wait(&ctl->empty[s], p.ph ^ 1u); if (!okw) { failed = true; return false; }
            }
            const uint32_t b_base = smem_u32(smem + s * kFwdStageBytes + 2 * kTileBytes);
#pragma unroll
            for (int r = 0; r < RPP; ++r) {
                const uint4 v = gather_finish_w<D, DEFORM>(p.q[r], p.w[r]);
                st_shared_v4(b_base + swz_offset(row0 + RS * (p.h * RPP + r), chunk), v.x, v.y, v.z, v.w);
            }
            if (p.h == PPS - 1) {
                fence_proxy_async_smem();
                mbar_arrive_warp(&ctl->full[s]);
            }
            return true;
        };
        if constexpr (kOverlap) {
            Pass pa, pb;
            bool ha = issue(pa);
            while (ha) {
                const bool hb = issue(pb);
                if (!finish(pa)) break;
                if (!hb) break;
                ha = issue(pa);
                if (!finish(pb)) break;
            }
        } else {
            Pass pa;
            while (issue(pa)) {
                if (!finish(pa)) break;
            }
        }
    }

    // teardown: every role has left its loop (normally or after a bounded wait gave up)
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// Largest number of distinct (deformable group, tap) keys any 64-wide K chunk touches.
inline int max_slots_per_chunk(const Geom& g, int cols_per_chunk) {
    const int kq = g.kv * g.Cg, width = cols_per_chunk * 8;
    int best = 1;
    if (g.Cg % g.cpg == 0 || g.cpg % g.Cg == 0) {          // keys change at every multiple of the segment length
        const int seg = g.cpg < g.Cg ? g.cpg : g.Cg;
        for (int k0 = 0; k0 < kq; k0 += width) {
            const int k1 = k0 + width < kq ? k0 + width : kq;
            const int slots = (k1 - 1) / seg - k0 / seg + 1 + (k0 + width > kq ? 1 : 0);
            if (slots > best) best = slots;
        }
        return best;
    }
    for (int j = 0; j < g.G; ++j) {
        for (int k0 = 0; k0 < kq; k0 += cols_per_chunk * 8) {
            int slots = 0, prev = -2;
            for (int c8 = 0; c8 < cols_per_chunk; ++c8) {
                const int kp = k0 + c8 * 8;
                int key = -1;
                if (kp < kq) {
                    const int tap = kp / g.Cg, cl = kp % g.Cg;
                    key = ((j * g.Cg + cl) / g.cpg) * g.kv + tap;
                }
                if (c8 == 0 || key != prev) ++slots;
                prev = key;
            }
            if (slots > best) best = slots;
        }
    }
    return best;
}

// The tiles' split along K, so that the SMs are busy to the end; both ways are weighed in K chunks of work (0.7 us each), an
// item costing six beside its own (set-up and epilogue), the fold four, and no item gets under three (B200, 2 x 128 channels
// 40x41, 26 tiles of 18 chunks, kernel time with reductions at 9 / 6 / 5 / 3 chunks an item: 18.3 / 15.6 / 14.8 / 13.9 us):
//   every tile into KS0 pieces (few tiles, or a badly filled last wave);
//   the R tiles left after the last full wave into KS1 pieces, as many as there are SMs to take them.
// room: bytes there are for slices; a split that needs more is not taken.
inline size_t fwd_slice_bytes(const Geom& g) { return (size_t)(g.Og > 128 ? 2 : 1) * kSliceHalf * sizeof(float); }
inline long long fwd_slices(const FwdSplit& sp) { return sp.KS0 > 1 ? sp.T0 : (sp.KS1 > 1 ? sp.n_items - sp.T0 : 0); }
inline FwdSplit fwd_split(const Geom& g, size_t room) {
    const TcDims d = tc_dims(g);
    const long long base_tiles = (long long)g.G * d.MB * d.PT;
    FwdSplit sp = {};
    sp.KS0 = sp.KS1 = 1;
    sp.cpk0 = sp.cpk1 = d.KC;
    sp.T0 = sp.tile1 = sp.n_items = base_tiles;
    if (base_tiles >= (1 << 28)) return sp;              // (the fold counts tiles and pieces in 32 bits)
    const int S = sm_count(), base = (int)base_tiles;
    const size_t most = room / fwd_slice_bytes(g);
    auto cost = [&](int items, int chunks) { return (items + S - 1) / S * (long long)(chunks + 6); };
    auto pieces = [&](int want, int& chunks) {           // of a tile; chunks: of one piece
        chunks = (d.KC + want - 1) / want;
        return (d.KC + chunks - 1) / chunks;
    };
    long long best = cost(base, d.KC);
    for (int k = 2; k <= d.KC / 3 && (long long)base * k <= 3ll * S; ++k) {
        int chunks;
        const int ks = pieces(k, chunks);
        const long long c = cost(base * ks, chunks) + 4;
        if (c * 20 < best * 19 && (size_t)base * ks <= most) { best = c; sp.KS0 = ks; sp.cpk0 = chunks; }
    }
    const int R = base % S;
    int ks1 = 1, cpk1 = d.KC;
    if (base > S && R != 0) {
        int want = S / R;
        if (want > d.KC / 3) want = d.KC / 3;
        if (want >= 2) {
            ks1 = pieces(want, cpk1);
            if ((long long)(base / S) * (d.KC + 6) + cost(R * ks1, cpk1) + 4 < best && (size_t)R * ks1 <= most) {
                sp.KS0 = 1;
                sp.cpk0 = d.KC;
            } else {
                ks1 = 1;
            }
        }
    }
    const bool tail = ks1 > 1;
    sp.T0 = tail ? base_tiles - R : base_tiles * sp.KS0;
    sp.tile1 = tail ? sp.T0 : base_tiles;
    sp.KS1 = ks1;
    sp.cpk1 = tail ? cpk1 : d.KC;
    sp.n_items = tail ? sp.T0 + R * ks1 : sp.T0;
    return sp;
}

// How a forward pass runs: stages and work split.
struct FwdPlan {
    FwdSplit sp;
    int stages, n_tabs, smem, max_slots, grid;
    int turn;                            // rows of a channel-first y are not 16-byte aligned
    bool direct;                         // the corner table does not fit beside the stages
    bool folds() const { return !direct && fwd_slices(sp) > 0; }
};

// accumulate: add to what y holds (the direct variant cannot)
template <int D, bool DEFORM>
FwdPlan fwd_plan(const Geom& g, const FwdSplit& split, const float* y, bool accumulate) {
    FwdPlan pl = {};
    pl.max_slots = max_slots_per_chunk(g, 8);
    pl.turn = !g.cl && (g.ov % 4 != 0 || (reinterpret_cast<uintptr_t>(y) & 15) != 0) ? 1 : 0;
    const size_t tab_one = (size_t)pl.max_slots * 128 * sizeof(TabEntry<D, DEFORM>);
    const size_t ost_bytes = (size_t)kFwdOffRing * pl.max_slots * D * 128 * sizeof(float);
    auto need = [&](int stages, int tabs) {
        return (long long)stages * kFwdStageBytes + (long long)tabs * tab_one + ost_bytes + sizeof(FwdCtl) + (pl.turn ? kFwdOutBytes : 0) + 1024;
    };
    // The four coordinate warps work on four tables at once and wait on the barriers of a table buffer by phase
    // parity, which is only sound while no warp runs two laps of the ring ahead of another: with the tables
    // consumed in order that holds for rings of four and more.  A ring of five or six comes before the fourth
    // operand stage (the stage count hardly matters: the producers, not the MMA, bound a stage).
    const int pref[][2] = {{4, 6}, {4, 5}, {3, 6}, {3, 5}, {4, 4}, {3, 4}, {2, 6}, {2, 5}, {2, 4}};
    for (const auto& c : pref) {
        if (need(c[0], c[1]) <= kSmemLimit) { pl.stages = c[0]; pl.n_tabs = c[1]; break; }
    }
    if (pl.stages == 0) {
        pl.direct = true;
        return pl;
    }
    pl.smem = (int)need(pl.stages, pl.n_tabs);
    pl.sp = split;
    pl.sp.acc = accumulate ? 1 : 0;
    pl.grid = (int)(pl.sp.n_items < sm_count() ? pl.sp.n_items : sm_count());
    return pl;
}

template <int D, bool DEFORM>
int launch_tc_forward(const Geom& g, const FwdPlan& pl, const __nv_bfloat16* xcl, const float* off, const uint8_t* wpk,
                      const float* bias, float* y, float* slices, cudaStream_t st) {
    if (pl.direct) return launch_tc_forward_direct<D, DEFORM>(g, xcl, off, wpk, bias, y, st);
    const TcDims d = tc_dims(g);
    constexpr int GW = 16;
    auto kern = pl.turn ? tc_forward_kernel<D, DEFORM, GW, true> : tc_forward_kernel<D, DEFORM, GW, false>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, pl.smem) != cudaSuccess) return -5;
    return launch_dependent(kern, dim3(pl.grid), dim3(fwd_threads(GW)), pl.smem, st, g, xcl, off, wpk, bias, y, d.KC, d.MT, d.MB,
                            d.PT, pl.stages, pl.max_slots, pl.n_tabs, pl.sp, slices) == cudaSuccess ? 0 : -5;
}

inline FwdPlan fwd_plan(const Geom& g, const FwdSplit& split, int ndim, int deform, const float* y, bool accumulate) {
    if (ndim == 2) return deform ? fwd_plan<2, true>(g, split, y, accumulate) : fwd_plan<2, false>(g, split, y, accumulate);
    return deform ? fwd_plan<3, true>(g, split, y, accumulate) : fwd_plan<3, false>(g, split, y, accumulate);
}
inline int launch_tc_forward(const Geom& g, const FwdPlan& pl, int ndim, int deform, const __nv_bfloat16* xcl,
                             const float* off, const uint8_t* wpk, const float* bias, float* y, float* slices, cudaStream_t st) {
    if (ndim == 2) return deform ? launch_tc_forward<2, true>(g, pl, xcl, off, wpk, bias, y, slices, st)
                                 : launch_tc_forward<2, false>(g, pl, xcl, off, wpk, bias, y, slices, st);
    return deform ? launch_tc_forward<3, true>(g, pl, xcl, off, wpk, bias, y, slices, st)
                  : launch_tc_forward<3, false>(g, pl, xcl, off, wpk, bias, y, slices, st);
}
// the fold of the split tiles' slices into y (`bias` and `y` of the launch)
inline FoldY y_fold(const Geom& g, const FwdPlan& pl, const float* slices, const float* bias, float* y) {
    const TcDims d = tc_dims(g);
    const bool tail = pl.sp.KS0 == 1;
    FoldY f = {};
    f.slices = slices; f.bias = bias; f.y = y;
    f.parts = tail ? pl.sp.KS1 : pl.sp.KS0;
    f.tiles = (unsigned)(fwd_slices(pl.sp) / f.parts);
    f.tile1 = tail ? (unsigned)pl.sp.tile1 : 0u;
    f.halves = g.Og > 128 ? 2 : 1;
    f.MB = d.MB;
    f.add = pl.sp.acc;
    f.d_PT.init((uint32_t)d.PT);
    return f;
}
inline int launch_y_fold(const Geom& g, const FwdPlan& pl, const float* slices, const float* bias, float* y, bool last,
                         cudaStream_t st) {
    if (!pl.folds()) return 0;
    const FoldY f = y_fold(g, pl, slices, bias, y);
    return launch_dependent(tc_fold_y_kernel, dim3(f.tiles, 16u * (unsigned)f.halves), dim3(kPassThreads), 0, st, g, f,
                            last ? 1 : 0) == cudaSuccess ? 0 : -5;
}
