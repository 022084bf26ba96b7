// Layout passes around the tensor-core kernels (included by dcn_tc.cu inside its anonymous namespace): everything that
// has to happen before the first contraction of a call goes out as ONE launch, everything after the last as another.
//
// A pass is a list of jobs, each a range of blocks: input copy, weight tiles, packed dy, sampling points, zero fills; or
// dX transpose, dW fold, bias-gradient fold, fold of a forward pass's partial sums.  The jobs of a list are independent of one another.  Each job moves its
// tensor once with coalesced accesses, so what is left to save at small and medium sizes is launches and the gaps
// between them: a batch-1 inference call spent 10 of its 32 us of GPU time and most of its 36 us of host time in four
// launches in front of the kernel, a layer step 28 launches (199 us busy, 237 us elapsed).
#pragma once



enum JobType { kJobCopyX, kJobCastX, kJobWeight, kJobPackDy, kJobPackDyCl, kJobPoints, kJobZero, kJobDx, kJobDw, kJobBias, kJobY };
// operand tiles a weight job cuts (see the kernels for who reads which)
enum WeightTiles {
    kTilesFwd,      // [G][MT][KC] 128 o x 64 k', k' = tap * Cg + c                          forward
    kTilesFlip,     // the same of the transposed convolution: rows c, k' = (kv-1-tap) * Og + o    plain input gradient
    kTilesBwd,      // [G][NB][OC] 256 k' x 64 o                                             backward data
    kTilesSlab      // [G][C/G/8][OC] kv * 8 rows (tap, channel of the slab) x 64 o           2-D backward data
};

struct Job {
    int type, gi;                    // gi: which of the list's geometries
    unsigned blocks;
    const void* src;
    void* dst;
    void* aux;                       // pack dy: partial sums for the bias gradient, [G][MT][128][PC]
    unsigned int* mx;                // raised to the bit pattern of the largest magnitude (null: not wanted)
    int a, b, c, d, e;
    size_t z, z2;
    FastDiv div;
};

constexpr int kMaxJobs = 12, kMaxGeoms = 3;
constexpr int kPassThreads = 256;
constexpr int kWeightSmem = 20 * 1024;       // of one weight job's block: ten blocks per SM stay resident

// Partial sums of the split tiles of a forward pass, as its epilogue stores them; see fold_y.
// Floats of a slice: [128-row half][lane quarter][16-position group][4 of them][lane][4].
constexpr int kSliceGroup = 4 * 32 * 4, kSliceHalf = 4 * (kTileN / 16) * kSliceGroup;
struct FoldY {
    const float *slices, *bias;
    float* y;
    unsigned tiles, tile1;           // split tiles, the first of them
    int parts, halves, MB, add;
    FastDiv d_PT;
};

struct JobList {
    Geom g[kMaxGeoms];
    Job job[kMaxJobs];
    FoldY fy;                        // of the kJobY job
    int n;
    int last;                        // no kernel of the call follows
};

// x [N, C, iv] fp32 -> [N, iv, C] bf16: tiles of 64 channels x 64 positions, sixteen loads of a thread in flight, 128-byte
// reads along the positions, 128-byte writes of bf16 pairs along the channels (C is a multiple of 8).
// a, b: tiles along positions / channels
__device__ __forceinline__ void job_copy_x(const Geom& g, const Job& J, unsigned blk, float* sm) {
    float (*tile)[65] = reinterpret_cast<float (*)[65]>(sm);
    const unsigned px = blk % J.a, r = blk / J.a, cy = r % J.b, n = r / J.b;
    const int p0 = (int)px * 64, c0 = (int)cy * 64, C = g.C, iv = g.iv;
    const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;
    const float* xn = static_cast<const float*>(J.src) + (size_t)n * C * iv;
    float v[2][8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int c = c0 + ty + i * 8;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int p = p0 + h * 32 + tx;
            v[h][i] = (c < C && p < iv) ? gload(xn + (size_t)c * iv + p) : 0.f;
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) tile[ty + i * 8][h * 32 + tx] = v[h][i];
    __syncthreads();
    uint32_t* on = reinterpret_cast<uint32_t*>(static_cast<__nv_bfloat16*>(J.dst) + (size_t)n * iv * C);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int q = ty + i * 8, p = p0 + q, c = c0 + 2 * tx;
        if (p < iv && c < C) on[((size_t)p * C + c) >> 1] = pack_bf16x2(tile[2 * tx][q], tile[2 * tx + 1][q]);
    }
}

// fp32 -> bf16 of an input that already is channels-last.  z: groups of 8 elements
__device__ __forceinline__ void job_cast_x(const Job& J, unsigned blk) {
    for (size_t i = (size_t)blk * kPassThreads + threadIdx.x; i < J.z; i += (size_t)J.blocks * kPassThreads) {
        const float4 a = gload(static_cast<const float4*>(J.src) + 2 * i);
        const float4 b = gload(static_cast<const float4*>(J.src) + 2 * i + 1);
        static_cast<uint4*>(J.dst)[i] = make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y),
                                                   pack_bf16x2(b.z, b.w));
    }
}

// W [O][Cg][kv] fp32 -> operand tiles, rounded once.  A block takes R output channels x a run of input channels (all
// taps: one contiguous piece of W per output channel) into shared memory and writes 16-byte chunks of tile rows; rows
// and columns of the tiles beyond the weight are written as zeros.
// a: WeightTiles, b: output channels per block, c: input channels per block, d: input-channel runs, e: output-channel runs
__device__ __forceinline__ void job_weight(const Geom& g, const Job& J, unsigned blk, float* sm) {
    const int R = J.b, CC = J.c, kv = g.kv;
    const int c0 = (int)(blk % J.d) * CC, ro = (int)(blk / J.d % J.e), j = (int)(blk / J.d / J.e), r0 = ro * R;
    const int nc = c0 >= g.Cg ? 0 : (g.Cg - c0 < CC ? g.Cg - c0 : CC);     // (flip: runs past the group pad the tile)
    const int stride = CC * kv + 1;
    const float* w = static_cast<const float*>(J.src);
    uint8_t* dst = static_cast<uint8_t*>(J.dst);
    if (J.aux != nullptr && blk == 0 && threadIdx.x == 0) *static_cast<unsigned int*>(J.aux) = 0u;
    float mx = 0.f;
#pragma unroll 4
    for (int e = threadIdx.x; e < R * CC * kv; e += kPassThreads) {        // (div: by CC * kv)
        uint32_t r, i;
        J.div.divmod((uint32_t)e, r, i);
        float v = 0.f;
        if (r0 + (int)r < g.Og && (int)i < nc * kv) v = gload(w + ((size_t)(j * g.Og + r0 + r) * g.Cg + c0) * kv + i);
        sm[r * stride + i] = v;
        mx = fmaxf(mx, fabsf(v));
    }
    if (J.mx != nullptr) {
        const unsigned int m = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
        if ((threadIdx.x & 31) == 0 && m != 0) atomicMax(J.mx, m);
    }
    __syncthreads();
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    const bool last = c0 + CC >= g.Cg;
    if (J.a == kTilesFwd) {
        const int MT = (g.Og + 127) / 128, KC = (g.Kg + 63) / 64, n8 = nc / 8, tail = last ? (KC * 64 - g.Kg) / 8 : 0;
        auto at = [&](int o, int kp) {
            return dst + (size_t)((j * MT + o / 128) * KC + kp / 64) * kTileBytes + swz_offset(o % 128, (kp % 64) / 8);
        };
        for (int e = threadIdx.x; e < R * kv * n8; e += kPassThreads) {
            const int c8 = e % n8, t = e / n8, tap = t % kv, r = t / kv;
            const float* s = sm + r * stride + c8 * 8 * kv + tap;
            if (r0 + r < MT * 128)
                *reinterpret_cast<uint4*>(at(r0 + r, tap * g.Cg + c0 + c8 * 8)) =
                    make_uint4(pack_bf16x2(s[0], s[kv]), pack_bf16x2(s[2 * kv], s[3 * kv]), pack_bf16x2(s[4 * kv], s[5 * kv]),
                               pack_bf16x2(s[6 * kv], s[7 * kv]));
        }
        for (int e = threadIdx.x; e < R * tail; e += kPassThreads)
            if (r0 + e / tail < MT * 128) *reinterpret_cast<uint4*>(at(r0 + e / tail, g.Kg + (e % tail) * 8)) = zero;
        return;
    }
    // the other tiles have eight output channels in a chunk; R = 64
    auto chunk = [&](int c, int tap, int o8) {
        const float* s = sm + o8 * 8 * stride + c * kv + tap;
        return make_uint4(pack_bf16x2(s[0], s[stride]), pack_bf16x2(s[2 * stride], s[3 * stride]),
                          pack_bf16x2(s[4 * stride], s[5 * stride]), pack_bf16x2(s[6 * stride], s[7 * stride]));
    };
    if (J.a == kTilesFlip) {
        const int MT = (g.Cg + 127) / 128, K = kv * g.Og, KC = (K + 63) / 64;
        auto at = [&](int c, int kp) {
            return dst + (size_t)((j * MT + c / 128) * KC + kp / 64) * kTileBytes + swz_offset(c % 128, (kp % 64) / 8);
        };
        for (int e = threadIdx.x; e < CC * kv * 8; e += kPassThreads) {
            const int o8 = e % 8, t = e / 8, tap = t % kv, c = t / kv;
            if (r0 + o8 * 8 < g.Og && c0 + c < MT * 128)
                *reinterpret_cast<uint4*>(at(c0 + c, (kv - 1 - tap) * g.Og + r0 + o8 * 8)) = chunk(c, tap, o8);
        }
        const int tail = ro == J.e - 1 ? (KC * 64 - K) / 8 : 0;
        for (int e = threadIdx.x; e < CC * tail; e += kPassThreads)
            if (c0 + e / tail < MT * 128) *reinterpret_cast<uint4*>(at(c0 + e / tail, K + (e % tail) * 8)) = zero;
        return;
    }
    const int OC = (g.Og + 63) / 64;
    if (J.a == kTilesBwd) {
        const int NB = (g.Kg + 255) / 256;
        auto at = [&](int kp, int o8) {
            return dst + (size_t)((j * NB + kp / 256) * OC + ro) * (2 * kTileBytes) + swz_offset(kp % 256, o8);
        };
        for (int e = threadIdx.x; e < nc * kv * 8; e += kPassThreads) {
            const int o8 = e % 8, t = e / 8, c = t % nc, tap = t / nc;
            *reinterpret_cast<uint4*>(at(tap * g.Cg + c0 + c, o8)) = chunk(c, tap, o8);
        }
        const int tail = last ? NB * 256 - g.Kg : 0;
        for (int e = threadIdx.x; e < tail * 8; e += kPassThreads) *reinterpret_cast<uint4*>(at(g.Kg + e / 8, e % 8)) = zero;
    } else {
        const int SL = g.Cg / 8;
        for (int e = threadIdx.x; e < nc * kv * 8; e += kPassThreads) {
            const int o8 = e % 8, t = e / 8, c = t % nc, tap = t / nc;
            *reinterpret_cast<uint4*>(dst + (size_t)((j * SL + (c0 + c) / 8) * OC + ro) * kv * 1024 +
                                      swz_offset(tap * 8 + (c0 + c) % 8, o8)) = chunk(c, tap, o8);
        }
    }
}

// dy [N, O, ov] fp32 -> bf16 tiles [G][MT][PC][128 o rows x 64 positions], swizzled; rows >= Og and positions >= P are
// zero.  Used by both backward kernels.  a: MT, z: PC; mx: max|dy|; aux: per-tile row sums
__device__ __forceinline__ void job_pack_dy(const Geom& g, const Job& J, unsigned blk, float* sm) {
    const long long PC = (long long)J.z;
    const long long pc = blk % (unsigned)PC;
    const int mt = (int)(blk / (unsigned)PC) % J.a, j = (int)(blk / (unsigned)PC) / J.a;
    const float* dy = static_cast<const float*>(J.src);
    uint8_t* dst = static_cast<uint8_t*>(J.dst) + (((size_t)j * J.a + mt) * PC + pc) * kTileBytes;
    const int lane = threadIdx.x % 32, wrp = threadIdx.x / 32;
    // lane handles positions 2*lane, 2*lane+1 of the 64; each warp walks rows wrp, wrp+8, ...
    const long long P0 = pc * 64 + 2 * lane;
    uint32_t n0 = 0, op0 = 0, n1 = 0, op1 = 0;
    const bool ok0 = P0 < g.P, ok1 = P0 + 1 < g.P;
    if (ok0) g.d_ov.divmod((uint32_t)P0, n0, op0);
    if (ok1) g.d_ov.divmod((uint32_t)(P0 + 1), n1, op1);
    float mx = 0.f;
    // both positions in one sample and 8-byte aligned (even ov, aligned dy): one 8-byte load per row
    const bool pair = ok1 && n0 == n1 && (g.ov & 1) == 0 && (reinterpret_cast<uintptr_t>(dy) & 7) == 0;
    const float* src0 = dy + ((size_t)n0 * g.O + (size_t)j * g.Og) * g.ov + op0;
    const float* src1 = dy + ((size_t)n1 * g.O + (size_t)j * g.Og) * g.ov + op1;
    for (int q = 0; q < 4; ++q) {
        float a[4], b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {                // four rows in flight
            const int ol = mt * 128 + wrp + (q * 4 + u) * 8;
            a[u] = b[u] = 0.f;
            if (ol < g.Og) {
                if (pair) {
                    const float2 t = gload(reinterpret_cast<const float2*>(src0 + (size_t)ol * g.ov));
                    a[u] = t.x; b[u] = t.y;
                } else {
                    if (ok0) a[u] = gload(src0 + (size_t)ol * g.ov);
                    if (ok1) b[u] = gload(src1 + (size_t)ol * g.ov);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int row = wrp + (q * 4 + u) * 8;
            mx = fmaxf(mx, fmaxf(fabsf(a[u]), fabsf(b[u])));
            const uint32_t ck = lane / 4;            // 8 positions per 16-byte chunk
            *reinterpret_cast<uint32_t*>(dst + swz_offset(row, ck) + (lane % 4) * 4) = pack_bf16x2(a[u], b[u]);
            if (J.aux != nullptr && mt * 128 + row < g.Og) {
                float s = a[u] + b[u];
#pragma unroll
                for (int m = 16; m >= 1; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
                if (lane == 0) static_cast<float*>(J.aux)[(((size_t)j * J.a + mt) * 128 + row) * PC + pc] = s;
            }
        }
    }
    if (J.mx != nullptr) {
        unsigned int* blk_max = reinterpret_cast<unsigned int*>(sm);
        if (threadIdx.x == 0) *blk_max = 0u;
        __syncthreads();
        const unsigned int m = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
        if (lane == 0 && m != 0) atomicMax(blk_max, m);
        __syncthreads();
        if (threadIdx.x == 0 && *blk_max != 0) atomicMax(J.mx, *blk_max);
    }
}

// Same tiles from a channels-last dy [N * ov positions][O]: a thread packs 8 consecutive positions of one output
// channel (one 16-byte chunk); consecutive threads take consecutive channels, so the reads coalesce.
__device__ __forceinline__ void job_pack_dy_cl(const Geom& g, const Job& J, unsigned blk, float* sm) {
    const long long PC = (long long)J.z;
    const long long pc = blk % (unsigned)PC;
    const int mt = (int)(blk / (unsigned)PC) % J.a, j = (int)(blk / (unsigned)PC) / J.a;
    const float* dy = static_cast<const float*>(J.src);
    uint8_t* dst = static_cast<uint8_t*>(J.dst) + (((size_t)j * J.a + mt) * PC + pc) * kTileBytes;
    const int row = threadIdx.x % 128;
    const int ol = mt * 128 + row;
    float sum = 0.f;
    for (int ck = threadIdx.x / 128; ck < 8; ck += kPassThreads / 128) {
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const long long P = pc * 64 + ck * 8 + e;
            v[e] = (ol < g.Og && P < g.P) ? gload(dy + (size_t)P * g.O + j * g.Og + ol) : 0.f;
            sum += v[e];
        }
        *reinterpret_cast<uint4*>(dst + swz_offset(row, ck)) =
            make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
    }
    if (J.aux != nullptr) {
        sm[threadIdx.x] = sum;
        __syncthreads();
        if (threadIdx.x < 128 && ol < g.Og)
            static_cast<float*>(J.aux)[(((size_t)j * J.a + mt) * 128 + row) * PC + pc] = sm[threadIdx.x] + sm[threadIdx.x + 128];
    }
}

// Sampling points of the 2-D backward-data kernel, located once for all channel slabs of a deformable group.  One
// 16-byte entry per (sample, deformable group, tap, output position), positions contiguous:
//   x  bits 0-19 byte offset of the (lo_h, lo_w) pixel in the blocked dX plane | bits 27-28 its class
//      | bit 29 hi_w != lo_w | bit 30 hi_h != lo_h | bit 31 valid
//   y  lo_h * Wp + lo_w (pixel index in the linear x plane)      z, w  the fractions lw_h, lw_w (fp32 bits)
// An invalid point has bits 29-31 and the fractions zero and names some pixel inside the plane (the tap's
// undeformed position, clamped): the kernel adds zeros there, and spreading those zeros over the plane keeps
// them from colliding on one address.
// The point is located exactly as everywhere else in the library (locate: int32 base + offset in one fp32
// rounding, validity, truncation, edge rule); dcn_debug_tc_points decodes these entries for the bit-exactness test.
// a: Wp, b: W2
__device__ __forceinline__ void job_points(const Geom& g, const Job& J, unsigned blk) {
    const int Wp = J.a, W2 = J.b;
    const float* off = static_cast<const float*>(J.src);
    constexpr int U = 4;                             // points of a thread in flight
    const long long total = (long long)g.N * g.dg * g.kv * g.ov;
    const long long e0 = blk * (long long)(U * kPassThreads) + threadIdx.x;
    float offv[U][2];
    OutPos op[U];
    uint32_t tap[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const long long e = e0 + u * kPassThreads < total ? e0 + u * kPassThreads : 0;
        uint32_t q1, pos, q2, n, grp;
        g.d_ov.divmod((uint32_t)e, q1, pos);
        g.d_kv.divmod(q1, q2, tap[u]);
        n = q2 / (uint32_t)g.dg;
        grp = q2 - n * (uint32_t)g.dg;
        op[u] = decompose_pos(g, (long long)n * g.ov + pos);
        const float* ob = offset_ptr<float, 2>(g, offset_block<float, 2>(g, off, (int)n), (int)grp, (int)tap[u], op[u]);
        offv[u][0] = gload(ob);
        offv[u][1] = gload(ob + g.ov);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const long long e = e0 + u * kPassThreads;
        if (e >= total) break;
        Pt<float, 2> s;
        locate_with<float, 2>(g, offv[u], (int)tap[u], op[u], s);
        uint4 r = make_uint4(0u, 0u, 0u, 0u);
        int h0, w0;
        if (s.valid) {
            h0 = s.lo[0];
            w0 = s.lo[1];
            r.x = ((s.hi[1] != w0 ? 1u : 0u) << 29) | ((s.hi[0] != h0 ? 1u : 0u) << 30) | (1u << 31);
            r.z = __float_as_uint(s.lw[0]);
            r.w = __float_as_uint(s.lw[1]);
        } else {
            h0 = op[u].base[1] < 0 ? 0 : (op[u].base[1] >= g.in[1] ? g.in[1] - 1 : op[u].base[1]);
            w0 = op[u].base[2] < 0 ? 0 : (op[u].base[2] >= g.in[2] ? g.in[2] - 1 : op[u].base[2]);
        }
        const uint32_t cls = (uint32_t)((h0 & 1) * 2 + (w0 & 1));
        r.x |= (uint32_t)(((h0 >> 1) * W2 + (w0 >> 1)) * 128) + cls * 32u + (cls << 27);
        r.y = (uint32_t)(h0 * Wp + w0);
        static_cast<uint4*>(J.dst)[e] = r;
    }
}

// Zero fill of z floats at dst and z2 floats at aux (16-byte stores where aligned).  b: blocks of the first range
constexpr int kZeroPerBlock = 16 * kPassThreads;
__device__ __forceinline__ void job_zero(const Job& J, unsigned blk) {
    const bool second = blk >= (unsigned)J.b;
    float* p = static_cast<float*>(second ? J.aux : J.dst);
    const size_t base = (size_t)(second ? blk - J.b : blk) * kZeroPerBlock, len = second ? J.z2 : J.z;
    const size_t n4 = (reinterpret_cast<uintptr_t>(p) & 15) == 0 ? len / 4 : 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const size_t e = base / 4 + i * kPassThreads + threadIdx.x;
        if (e < n4) {
            reinterpret_cast<float4*>(p)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (e * 4 + k < len) p[e * 4 + k] = 0.f;
        }
    }
}

// dx[n, c, p] (+)= dx_cl[n, p, c], tiles of 64 x 64.  a, b: tiles along positions / channels; c: add
__device__ __forceinline__ void job_dx(const Geom& g, const Job& J, unsigned blk, float* sm) {
    float (*tile)[65] = reinterpret_cast<float (*)[65]>(sm);
    const unsigned px = blk % J.a, r = blk / J.a, cy = r % J.b, n = r / J.b;
    const int p0 = (int)px * 64, c0 = (int)cy * 64, C = g.C, iv = g.iv;
    const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;
    const float* in = static_cast<const float*>(J.src) + (size_t)n * iv * C;
    float v[2][8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int p = p0 + ty + i * 8;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = c0 + h * 32 + tx;
            v[h][i] = (p < iv && c < C) ? gload(in + (size_t)p * C + c) : 0.f;
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) tile[ty + i * 8][h * 32 + tx] = v[h][i];
    __syncthreads();
    float* out = static_cast<float*>(J.dst) + (size_t)n * C * iv;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int cl = ty + i * 8, c = c0 + cl;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int p = p0 + h * 32 + tx;
            if (c < C && p < iv) {
                if (J.c) out[(size_t)c * iv + p] += tile[h * 32 + tx][cl];
                else out[(size_t)c * iv + p] = tile[h * 32 + tx][cl];
            }
        }
    }
}

// dwpk[split][k' / 4][rows][4] (k' = tap * Cg + c) -> dW [O][Cg][kv], the position splits added in split order
// (deterministic).  A block takes 8 output channels, 32 input channels and a run of up to 4 taps, one 16-byte vector of
// channels per thread and split: slices read along the rows (128-byte runs), dW written along the taps.
// a: rows of a group, c: add, d: splits, e: channel runs; z: slice elements, z2: tap runs
constexpr int kFoldChannels = 32, kFoldRows = 8, kFoldTaps = 4;
__device__ __forceinline__ void job_dw(const Geom& g, const Job& J, unsigned blk, float* sm) {
    const int kv = g.kv, runs = (int)J.z2, per = (kv + runs - 1) / runs, orun = (g.Og + kFoldRows - 1) / kFoldRows;
    const int t0 = (int)(blk % runs) * per, c0 = (int)(blk / runs % J.e) * kFoldChannels;
    const int ro = (int)(blk / runs / J.e), j = ro / orun, o0 = (ro - j * orun) * kFoldRows;
    const int nc = g.Cg - c0 < kFoldChannels ? g.Cg - c0 : kFoldChannels, nt = kv - t0 < per ? kv - t0 : per;
    const int r = threadIdx.x % kFoldRows, c4 = threadIdx.x / kFoldRows % (kFoldChannels / 4), t = threadIdx.x / (2 * kFoldChannels);
    if (o0 + r < g.Og && c4 * 4 < nc && t < nt) {
        const size_t rows = (size_t)g.G * J.a;
        const float4* s = static_cast<const float4*>(J.src) + (size_t)(((t0 + t) * g.Cg + c0) / 4 + c4) * rows + j * J.a + o0 + r;
        // loads in batches of four (independent, all in flight), additions in split order
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int s0 = 0; s0 < J.d; s0 += 4) {
            float4 q[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) q[u] = (s0 + u < J.d) ? gload(s + (size_t)(s0 + u) * (J.z / 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int u = 0; u < 4; ++u) { v.x += q[u].x; v.y += q[u].y; v.z += q[u].z; v.w += q[u].w; }
        }
        float* d = sm + (r * kFoldChannels + c4 * 4) * (kFoldTaps + 1) + t;
        d[0] = v.x; d[kFoldTaps + 1] = v.y; d[2 * (kFoldTaps + 1)] = v.z; d[3 * (kFoldTaps + 1)] = v.w;
    }
    __syncthreads();
    const int rn = g.Og - o0 < kFoldRows ? g.Og - o0 : kFoldRows;
    for (int e = threadIdx.x; e < rn * nc * nt; e += kPassThreads) {
        const int wt = e % nt, q = e / nt, wc = q % nc, wr = q / nc;
        float* d = static_cast<float*>(J.dst) + ((size_t)(j * g.Og + o0 + wr) * g.Cg + c0 + wc) * kv + t0 + wt;
        const float v = sm[(wr * kFoldChannels + wc) * (kFoldTaps + 1) + wt];
        *d = J.c ? *d + v : v;
    }
}

// dbias[o] = sum over the dy tiles of a row, one warp per output channel.  a: MT, z: PC
__device__ __forceinline__ void job_bias(const Geom& g, const Job& J, unsigned blk) {
    const int o = (int)blk * (kPassThreads / 32) + threadIdx.x / 32, lane = threadIdx.x % 32;
    if (o >= g.O) return;
    const int j = o / g.Og, ol = o - j * g.Og;
    const float* s = static_cast<const float*>(J.src) + ((size_t)j * J.a * 128 + ol) * J.z;
    float v = 0.f;
    for (size_t i = lane; i < J.z; i += 32) v += gload(s + i);
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
    if (lane == 0) static_cast<float*>(J.dst)[o] = v;
}

// y of the split tiles of a forward pass: the slices of a tile added in K order, plus the bias.  (Reductions into a zeroed y
// left the order, and with it the last bits, to whichever part came first.)  A block takes 32 output channels x 32 positions,
// one 16-byte vector of every slice per thread, in the order in which the epilogue stored them; y leaves in 128-byte runs,
// along the positions or the channels.
// Bound by latency (launch, one read of L2, one turn).  Against the reductions, B200: one image 256 -> 256 channels 50x76,
// 30 tiles in 4 parts: kernel 26.3 -> 20.0 us and 4.2 us of fold, call 28.2 -> 28.5; 8 x 128 -> 128, 28x28 as a layer, three
// forward kernels in 3 parts: step 142 -> 150 us; config 2, 44 of 784 tiles in 3 parts: 1210 -> 1214.  Folding in the CTA that finishes a tile last is slower: its
// slices then pass through one SM (kernel 34.6 us for the first, step 170 us for the second).
// piece: [half][lane quarter][32 positions]
__device__ __forceinline__ void fold_y(const Geom& g, const FoldY& a, unsigned slot, unsigned piece, float* sm) {
    const int cg = (int)(piece % 4), q = (int)(piece / 4 % 4), mt = (int)(piece / 16);
    uint32_t jm, pt;
    a.d_PT.divmod(a.tile1 + slot, jm, pt);
    const int j = (int)(jm / (unsigned)a.MB), mb = (int)jm - j * a.MB;
    const int o0 = (mb * 2 + mt) * 128 + q * 32, lane = threadIdx.x % 32, wp = threadIdx.x / 32;
    const long long P0 = (long long)pt * kTileN + cg * 32;
    if (o0 >= g.Og || P0 >= g.P) return;
    const size_t step = (size_t)a.halves * kSliceHalf / 4;
    const float4* s = reinterpret_cast<const float4*>(a.slices) + (size_t)slot * a.parts * step +
                      (mt * kSliceHalf + q * (kSliceHalf / 4) + cg * 2 * kSliceGroup) / 4 + threadIdx.x;
    const float bv = a.bias != nullptr && o0 + lane < g.Og ? gload(a.bias + j * g.Og + o0 + lane) : 0.f;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k0 = 0; k0 < a.parts; k0 += 4) {    // loads in batches of four (all in flight), additions in order
        float4 t[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) t[u] = k0 + u < a.parts ? gload(s + (k0 + u) * step) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 4; ++u) { v.x += t[u].x; v.y += t[u].y; v.z += t[u].z; v.w += t[u].w; }
    }
    float* row = sm + lane * 33 + wp * 4;        // positions 4 * wp .. of channel `lane`
    row[0] = v.x + bv; row[1] = v.y + bv; row[2] = v.z + bv; row[3] = v.w + bv;
    __syncthreads();
    const int o = j * g.Og + o0;
    if (g.cl) {
        float* d = a.y + (size_t)(P0 + wp) * g.O + o + lane;
#pragma unroll
        for (int i = 0; i < 4; ++i, d += 8 * (size_t)g.O) {
            if (o0 + lane >= g.Og || P0 + wp + 8 * i >= g.P) continue;
            const float r = sm[lane * 33 + wp + 8 * i];
            *d = a.add ? *d + r : r;
        }
    } else if (P0 + lane < g.P) {
        uint32_t n, opos;
        g.d_ov.divmod((uint32_t)P0 + lane, n, opos);
        float* d = a.y + ((size_t)n * g.O + o + wp) * g.ov + opos;
#pragma unroll
        for (int i = 0; i < 4; ++i, d += 8 * (size_t)g.ov) {
            if (o0 + wp + 8 * i >= g.Og) continue;
            const float r = sm[(wp + 8 * i) * 33 + lane];
            *d = a.add ? *d + r : r;
        }
    }
}

// behind a forward pass, a launch of its own: grid (tiles, pieces).  last: no kernel of the call follows
__global__ void __launch_bounds__(kPassThreads)
tc_fold_y_kernel(const __grid_constant__ Geom g, const __grid_constant__ FoldY a, const int last) {
    __shared__ float sm[32 * 33];
    if (!last) pdl_trigger();
    pdl_wait();
    fold_y(g, a, blockIdx.x, blockIdx.y, sm);
}

__global__ void __launch_bounds__(kPassThreads, 6)
tc_passes_kernel(const __grid_constant__ JobList L) {
    extern __shared__ float pass_smem[];
    if (!L.last) pdl_trigger();
    pdl_wait();
    unsigned b = blockIdx.x;
    int i = 0;
    while (b >= L.job[i].blocks) b -= L.job[i++].blocks;
    const Job& J = L.job[i];
    const Geom& g = L.g[J.gi];
    switch (J.type) {
        case kJobCopyX: job_copy_x(g, J, b, pass_smem); break;
        case kJobCastX: job_cast_x(J, b); break;
        case kJobWeight: job_weight(g, J, b, pass_smem); break;
        case kJobPackDy: job_pack_dy(g, J, b, pass_smem); break;
        case kJobPackDyCl: job_pack_dy_cl(g, J, b, pass_smem); break;
        case kJobPoints: job_points(g, J, b); break;
        case kJobZero: job_zero(J, b); break;
        case kJobDx: job_dx(g, J, b, pass_smem); break;
        case kJobDw: job_dw(g, J, b, pass_smem); break;
        case kJobBias: job_bias(g, J, b); break;
        default: fold_y(g, L.fy, b / (unsigned)J.a, b % (unsigned)J.a, pass_smem); break;
    }
}

// Builder of one launch.  Jobs with no blocks are dropped; an error (misaligned pointer) is kept for launch().
class Passes {
public:
    Passes() { L.n = 0; }

    void copy_x(const Geom& g, const float* x, __nv_bfloat16* xcl) {
        if (g.cl) {
            if ((reinterpret_cast<uintptr_t>(x) & 15) != 0) { error = -7; return; }      // vector loads
            Job& J = add(g, kJobCastX, x, xcl);
            J.z = (size_t)g.N * g.iv * g.C / 8;
            const size_t want = (J.z + kPassThreads - 1) / kPassThreads;
            J.blocks = (unsigned)(want < (size_t)(8 * sm_count()) ? want : (size_t)(8 * sm_count()));
        } else {
            Job& J = add(g, kJobCopyX, x, xcl);
            J.a = (g.iv + 63) / 64;
            J.b = (g.C + 63) / 64;
            J.blocks = (unsigned)J.a * (unsigned)J.b * (unsigned)g.N;
            need(64 * 65 * 4);
        }
    }
    // clear: a word to set to zero on the way
    void weight(const Geom& g, WeightTiles tiles, const float* w, void* dst, unsigned int* mx = nullptr, unsigned int* clear = nullptr) {
        Job& J = add(g, kJobWeight, w, dst);
        J.mx = mx;
        J.aux = clear;
        J.a = tiles;
        int rows = g.Og, chans = g.Cg;
        if (tiles == kTilesFwd) {
            J.c = 64;
            while (J.c > 8 && J.c * g.kv * 4 > kWeightSmem) J.c /= 2;
            J.b = kWeightSmem / (J.c * g.kv * 4);
            J.b = J.b < 1 ? 1 : (J.b > 8 ? 8 : J.b);
            rows = (g.Og + 127) / 128 * 128;
        } else {
            J.b = 64;
            J.c = 8;
            while (J.c > 1 && 64 * J.c * g.kv * 4 > kWeightSmem) J.c /= 2;
            if (tiles == kTilesFlip) chans = (g.Cg + 127) / 128 * 128;
        }
        J.div.init((uint32_t)(J.c * g.kv));
        J.d = (chans + J.c - 1) / J.c;
        J.e = (rows + J.b - 1) / J.b;
        J.blocks = (unsigned)J.d * (unsigned)J.e * (unsigned)g.G;
        need(J.b * (J.c * g.kv + 1) * 4);
    }
    void pack_dy(const Geom& g, const float* dy, uint8_t* dpk, int MT, long long PC, unsigned int* mx, float* row_sums) {
        Job& J = add(g, g.cl ? kJobPackDyCl : kJobPackDy, dy, dpk);
        J.a = MT;
        J.z = (size_t)PC;
        J.mx = mx;
        J.aux = row_sums;
        J.blocks = (unsigned)PC * (unsigned)(g.G * MT);
        need(kPassThreads * 4);
    }
    void points(const Geom& g, const float* off, uint4* pts, int Wp, int W2) {
        Job& J = add(g, kJobPoints, off, pts);
        J.a = Wp;
        J.b = W2;
        J.blocks = (unsigned)(((long long)g.N * g.dg * g.kv * g.ov + 4 * kPassThreads - 1) / (4 * kPassThreads));
    }
    void zero(float* p, size_t len) {
        if (p == nullptr || len == 0) return;
        const unsigned blocks = (unsigned)((len + kZeroPerBlock - 1) / kZeroPerBlock);
        if (L.n > 0) {                                 // beside another one in the same job
            Job& last = L.job[L.n - 1];
            if (last.type == kJobZero && last.aux == nullptr) {
                last.aux = p;
                last.z2 = len;
                last.blocks += blocks;
                return;
            }
        }
        Job& J = add(L.g[0], kJobZero, nullptr, p);
        J.z = len;
        J.b = (int)blocks;
        J.blocks = blocks;
    }
    void fold_dx(const Geom& g, const float* dxcl, float* dx, bool add_to) {
        Job& J = add(g, kJobDx, dxcl, dx);
        J.a = (g.iv + 63) / 64;
        J.b = (g.C + 63) / 64;
        J.c = add_to ? 1 : 0;
        J.blocks = (unsigned)J.a * (unsigned)J.b * (unsigned)g.N;
        need(64 * 65 * 4);
    }
    void fold_dw(const Geom& g, const float* dwpk, float* dw, int rows, int splits, size_t slice, bool add_to) {
        Job& J = add(g, kJobDw, dwpk, dw);
        J.a = rows;
        J.c = add_to ? 1 : 0;
        J.d = splits;
        J.e = (g.Cg + kFoldChannels - 1) / kFoldChannels;
        J.z = slice;
        J.z2 = (size_t)(g.kv + kFoldTaps - 1) / kFoldTaps;
        J.blocks = (unsigned)(g.G * ((g.Og + kFoldRows - 1) / kFoldRows)) * (unsigned)J.e * (unsigned)J.z2;
        need(kFoldRows * kFoldChannels * (kFoldTaps + 1) * 4);
    }
    void fold_bias(const Geom& g, const float* row_sums, float* dbias, int MT, long long PC) {
        Job& J = add(g, kJobBias, row_sums, dbias);
        J.a = MT;
        J.z = (size_t)PC;
        J.blocks = (unsigned)((g.O + kPassThreads / 32 - 1) / (kPassThreads / 32));
    }

    // (one per launch)
    void fold_y(const Geom& g, const FoldY& f) {
        Job& J = add(g, kJobY, f.slices, f.y);
        J.a = 16 * f.halves;
        J.blocks = f.tiles * (unsigned)J.a;
        L.fy = f;
        need(32 * 33 * 4);
    }

    // one launch; last: of the call
    int launch(cudaStream_t st, bool last) {
        if (error != 0) return error;
        L.last = last ? 1 : 0;
        return L.n == 0 ? 0 : submit(L, st);
    }

private:
    JobList L;
    int smem = 0, error = 0, geoms = 0;
    const Geom* seen[kMaxGeoms] = {};

    void need(int bytes) { if (bytes > smem) smem = bytes; }
    Job& add(const Geom& g, int type, const void* src, void* dst) {
        int gi = 0;
        if (type != kJobZero) {
            while (gi < geoms && seen[gi] != &g) ++gi;
            if (gi == kMaxGeoms) { gi = 0; error = -5; }
            if (gi == geoms) { seen[gi] = &g; L.g[gi] = g; ++geoms; }
        }
        if (L.n == kMaxJobs) { error = -5; --L.n; }
        Job& J = L.job[L.n++];
        J = Job{};
        J.type = type; J.gi = gi; J.src = src; J.dst = dst;
        return J;
    }
    int submit(const JobList& l, cudaStream_t st) {
        unsigned long long blocks = 0;
        for (int i = 0; i < l.n; ++i) blocks += l.job[i].blocks;
        if (blocks == 0) return 0;
        if (blocks >= (1ull << 31)) return -8;
        if (smem > 48 * 1024 &&
            cudaFuncSetAttribute(tc_passes_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
            return -5;
        return launch_dependent(tc_passes_kernel, dim3((unsigned)blocks), dim3(kPassThreads), smem, st, l) == cudaSuccess ? 0 : -5;
    }
};
