// Fused kernels of the surrogate MLP for hidden = 256 and at most 32 inputs (the network the
// assimilation uses): the whole forward pass, and the backward pass through both hidden layers,
// in one kernel per 128-row tile; the weight gradients in a second one.
//
// The layer-by-layer kernels were bound by operand staging and passes over memory: the forward of
// 11,520 rows took 120 us for 1.6 GFLOP (two tensor-core GEMMs of 37 us, a one-column GEMM of 45).
// Here the activations of a tile stay in TMEM and shared memory: the accumulators of both layers
// (2 x 256 columns) fill TMEM, each hidden layer's GELU is applied as the accumulator is read, and
// the result is written straight into the next GEMM's operand buffer in 64-column chunks, the MMAs of
// one chunk running while the warps compute the next.  What bounds the forward is the elementwise
// work (erff and the three-term split, about 60 instructions per hidden unit): issue slots 57 % busy
// with two warps a scheduler, ALU pipe 45 %, tensor pipe 22 % (ncu, on the 90 SMs it uses); training
// waits on activation stores and reloads as well, the weight gradients on their loads.
// Measured: forward of 11,520 rows 120.3 -> 18.4 us, gradient of 4,096 rows 367 -> 84 us, an Adam
// step on 360 rows 375 -> 50 us; the error of the gradient against 64 bits 1.5e-6 -> 0.8e-6.
//
// Weights are read as BF16 "images" in the canonical shared-memory operand order (8 x 16-byte core
// matrices), written once when the weights change, so that a whole 256 x 256 operand arrives with
// one bulk copy.  FP32 operands enter as three BF16 terms, as in k_mma_gemm.
//
// Included by dtb_mlp.cu inside its anonymous namespace.

constexpr int kNetH = 256;                 // hidden units
constexpr int kNetMaxIn = 32;              // inputs, padded to 16 or 32
constexpr int kNetRows = 128;              // rows per CTA (tcgen05 M)
constexpr int kNetSMs = 148;               // SMs: one CTA each
constexpr int kNetThreads = 256;           // warp w: TMEM lanes 32 (w % 4).., column half w / 4
constexpr int kNetChunk = 64;              // hidden units per operand chunk
constexpr int kNetChunks = kNetH / kNetChunk;
constexpr int kNetTermBytes = kNetRows * kNetChunk * 2;           // one BF16 term of a chunk
constexpr int kNetW2Bytes = kNetH * kNetH * 2;
constexpr int kNetImgW2 = kNetH * kNetH;                           // elements
constexpr int kNetTmemCols = 512;
constexpr uint32_t kNetWait = 1u << 22;   // polls of a wait before it is given up (dtb_mlp_set_wait_limit)
constexpr uint32_t kNetDrain = 1u << 24;  // ... of the copies and MMAs still in flight at the end

// Element (row, k) of a K-major operand image of R rows: core matrices of 8 rows x 8 k (128 bytes),
// row groups adjacent, K groups R / 8 core matrices apart.
__host__ __device__ __forceinline__ int net_img(int R, int row, int k)
{
    return (((k >> 3) * (R >> 3) + (row >> 3)) << 6) + ((row & 7) << 3) + (k & 7);
}

// Shared-memory matrix descriptor: leading (K) and stride (8-row) byte offsets, no swizzle.
__device__ __forceinline__ uint64_t net_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((saddr >> 4) & 0x3fffu) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}

__device__ __forceinline__ void net_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool acc)
{
    const uint32_t p = acc ? 1u : 0u;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 :: "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(p) : "memory");
}

__device__ __forceinline__ void net_commit(uint32_t mbar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(mbar) : "memory");
}

__device__ __forceinline__ void net_ld16(uint32_t taddr, float* v)
{
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// C consecutive accumulator columns of the thread's lane (C = 8, 16 or 32).
template <int C>
__device__ __forceinline__ void net_ld(uint32_t taddr, float* v)
{
    if (C == 8) {
        uint32_t r[8];
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(taddr) : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
    } else {
#pragma unroll
        for (int c = 0; c < C; c += 16) net_ld16(taddr + (uint32_t)c, v + c);
    }
}

template <int C>
__device__ __forceinline__ void net_store(float* dst, const float* v)
{
#pragma unroll
    for (int e = 0; e < C; e += 4) *reinterpret_cast<float4*>(dst + e) = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
}

__device__ __forceinline__ void net_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t mbar)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(mbar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(dst), "l"(src), "r"(bytes), "r"(mbar) : "memory");
}

// Eight FP32 values as three BF16 terms (hi + mid + lo), one 16-byte store each.
// dup > 1: also `dup_bytes` further on, and so on (the copies of a row in the other quadrants).
__device__ __forceinline__ void net_split8(const float* x, unsigned char* dst, int term_bytes, int dup = 1, int dup_bytes = 0)
{
    uint32_t t[3][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        float a = x[2 * e], b = x[2 * e + 1];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
            t[i][e] = *reinterpret_cast<const uint32_t*>(&h);
            a -= __uint_as_float(t[i][e] << 16);
            b -= __uint_as_float(t[i][e] & 0xffff0000u);
        }
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
        for (int d = 0; d < dup; ++d)
            *reinterpret_cast<uint4*>(dst + i * term_bytes + d * dup_bytes) = make_uint4(t[i][0], t[i][1], t[i][2], t[i][3]);
}

// What was given up on lands before its shared memory and TMEM go (out of line: rarely run, and the
// kernels' loops are long enough for the instruction cache to notice).
__device__ __noinline__ void net_drain(uint32_t mbar, uint32_t parity) { mma_wait(mbar, parity, kNetDrain); }

struct NetArgs {
    int in, kx;                            // inputs, padded K of layer 1
    int64_t B;
    const float* x;                        // [B][in]
    const float* target;                   // [B] (training)
    const __nv_bfloat16* img1;             // W1 as [256][kx]
    const __nv_bfloat16* img2;             // W2 as B operand of layer 2 (rows o, K = i)
    const __nv_bfloat16* img2t;            // W2 as B operand of the backward pass (rows i, K = o)
    const float *b1, *b2, *b3;
    const __nv_bfloat16* w3;
    float* y;
    float *Z1, *H1, *H2, *dZ2, *dZ1, *dY;  // [B][256] (training), dY [B]
    float* loss;
    unsigned* err;
    uint32_t wait;                         // polls of a wait before it is given up
};

constexpr int kNetOffA = kNetW2Bytes;                               // the chunk's three terms
constexpr int kNetOffX = kNetOffA + 3 * kNetTermBytes;
constexpr int kNetOffW1 = kNetOffX + 3 * kNetRows * kNetMaxIn * 2;
constexpr int kNetOffF = kNetOffW1 + kNetH * kNetMaxIn * 2;         // b1, b2, w3 [256], partial y [2 D][128 / D], dy
constexpr int kNetSmem = kNetOffF + (3 * kNetH + 3 * kNetRows) * 4;
static_assert(kNetSmem <= 227 * 1024, "shared memory of one CTA");

// D: a CTA takes 128 / D rows, each of them D times in the tile (in D of the four TMEM quadrants,
// 32 lanes each, that a warp can read): the copies cost nothing on the tensor cores, and the warps of
// the D quadrants share a row's columns, so that a batch too small to fill the GPU with 128-row tiles
// spends 1 / D of the time on the elementwise work that bounds it (gradient of 4,096 rows 124 -> 87 us,
// Adam step on 360 rows 92 -> 54 us against D = 1).
// Once a wait was given up on, in any thread: y and dY of the CTA's rows and the loss become NaN, and
// the error flag keeps Adam from using what was not computed.  (Told to all at the barrier before the
// output and at the end; at every chunk's barrier it cost the forward of 11,520 rows 0.3 us more.)
template <bool TRAIN, int D>
__global__ void __launch_bounds__(kNetThreads, 1) k_net(NetArgs g)
{
    constexpr int kRows = kNetRows / D;
    constexpr int kQuads = 4 / D;                         // quadrants of distinct rows
    constexpr int kCols = kNetChunk / (2 * D);            // columns of a chunk per thread
    extern __shared__ __align__(1024) unsigned char nsm[];
    __shared__ __align__(8) unsigned long long bars[4];   // W1, W2, layer 1, chunk
    __shared__ uint32_t tmem_base;
    unsigned char* sW2 = nsm;
    unsigned char* sA = nsm + kNetOffA;
    unsigned char* sX = nsm + kNetOffX;
    unsigned char* sW1 = nsm + kNetOffW1;
    float* sb1 = reinterpret_cast<float*>(nsm + kNetOffF);
    float* sb2 = sb1 + kNetH;
    float* sw3 = sb2 + kNetH;
    float* sy = sw3 + kNetH;
    float* sdy = sy + 2 * kNetRows;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int quad = warp & 3;
    const int r = (quad % kQuads) * 32 + lane;            // tile row (its first copy)
    const int grp = (quad / kQuads) * 2 + (warp >> 2);    // the thread's share of a row's columns, 0 .. 2 D - 1
    const int64_t row = (int64_t)blockIdx.x * kRows + r;
    const bool live = row < g.B;
    const uint32_t b_w1 = smem_addr(&bars[0]), b_w2 = smem_addr(&bars[1]), b_l1 = smem_addr(&bars[2]), b_ch = smem_addr(&bars[3]);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_addr(&tmem_base)), "r"((uint32_t)kNetTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_addr(&bars[i])) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        net_bulk(smem_addr(sW1), g.img1, (uint32_t)(kNetH * g.kx * 2), b_w1);
        net_bulk(smem_addr(sW2), g.img2, (uint32_t)kNetW2Bytes, b_w2);
    }
    sb1[tid] = g.b1[tid];
    sb2[tid] = g.b2[tid];
    sw3[tid] = __bfloat162float(g.w3[tid]);
    // X: the thread's row, K groups grp, grp + 2 D, ... in three terms
    const int xterm = kNetRows * g.kx * 2;
    for (int c = grp; c < g.kx / 8; c += 2 * D) {
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int k = c * 8 + e;
            v[e] = (live && k < g.in) ? __ldg(g.x + row * g.in + k) : 0.0f;
        }
        net_split8(v, sX + (c * (kNetRows / 8) + (r >> 3)) * 128 + (r & 7) * 16, xterm, D, kRows * 16);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;
    const uint32_t tlane = tmem + ((uint32_t)(quad * 32) << 16);
    const uint32_t idesc = mma_idesc(kNetH);
    bool ok = true;
    bool l1 = false, w2t = false;   // thread 0: committed to b_l1; copy of W2^T issued
    int n_ch = 0;                   // thread 0: commits to b_ch
    if (tid == 0 && (ok = mma_wait(b_w1, 0, g.wait))) {   // layer 1: Z1 = X W1^T
        for (int s = 0; s < g.kx / 16; ++s)
            for (int i = 0; i < 3; ++i)
                net_mma(tmem, net_desc(smem_addr(sX + i * xterm + s * 2 * (kNetRows / 8) * 128), (kNetRows / 8) * 128, 128),
                        net_desc(smem_addr(sW1 + s * 2 * (kNetH / 8) * 128), (kNetH / 8) * 128, 128), idesc, s + i > 0);
        net_commit(b_l1);
        l1 = true;
    }
    ok = ok && mma_wait(b_l1, 0, g.wait);
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    // One operand chunk: the thread's kCols values of chunk q's columns into the buffer once the MMAs
    // that read the chunk before are done, then this chunk's MMAs into accumulator columns d (first: q == q0).
    auto chunk = [&](int q, int q0, uint32_t d, const float* v) {
        if (q >= 1) ok = ok && mma_wait(b_ch, (uint32_t)((q - 1) & 1), g.wait);
#pragma unroll
        for (int c = 0; c < kCols / 8; ++c)
            net_split8(v + c * 8, sA + ((grp * (kCols / 8) + c) * (kNetRows / 8) + (r >> 3)) * 128 + (r & 7) * 16, kNetTermBytes,
                       D, kRows * 16);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (tid == 0 && ok) {   // (so that at most one commit is outstanding when a wait is given up)
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int k8 = (q - q0) * (kNetChunk / 8);
            for (int s = 0; s < kNetChunk / 16; ++s)
                for (int i = 0; i < 3; ++i)
                    net_mma(d, net_desc(smem_addr(sA + i * kNetTermBytes + s * 2 * (kNetRows / 8) * 128), (kNetRows / 8) * 128, 128),
                            net_desc(smem_addr(sW2 + (k8 + 2 * s) * (kNetH / 8) * 128), (kNetH / 8) * 128, 128), idesc,
                            q > q0 || s + i > 0);
            net_commit(b_ch);
            ++n_ch;
        }
    };

    // ---- layer 2: Z2 = GELU(Z1 + b1) W2^T, chunk by chunk
    if (tid == 0) ok = ok && mma_wait(b_w2, 0, g.wait);
    for (int q = 0; q < kNetChunks; ++q) {
        float v[kCols];
        const int c0 = q * kNetChunk + grp * kCols;
        net_ld<kCols>(tlane + (uint32_t)c0, v);
#pragma unroll
        for (int e = 0; e < kCols; ++e) v[e] += sb1[c0 + e];
        if (TRAIN && live && ok) net_store<kCols>(g.Z1 + row * kNetH + c0, v);
#pragma unroll
        for (int e = 0; e < kCols; ++e) v[e] = gelu(v[e]);
        if (TRAIN && live && ok) net_store<kCols>(g.H1 + row * kNetH + c0, v);
        chunk(q, 0, tmem + kNetH, v);
    }
    ok = ok && mma_wait(b_ch, (uint32_t)((kNetChunks - 1) & 1), g.wait);
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (TRAIN && tid == 0 && ok) {
        net_bulk(smem_addr(sW2), g.img2t, (uint32_t)kNetW2Bytes, b_w2);   // every MMA that read W2 is done
        w2t = true;
    }

    // ---- output: y = GELU(Z2 + b2) . w3 + b3
    float p = 0.0f;
    for (int q = 0; q < kNetChunks; ++q) {
        float v[kCols];
        const int c0 = q * kNetChunk + grp * kCols;
        net_ld<kCols>(tlane + (uint32_t)(kNetH + c0), v);
#pragma unroll
        for (int e = 0; e < kCols; ++e) {
            v[e] = gelu(v[e] + sb2[c0 + e]);
            p = fmaf(v[e], sw3[c0 + e], p);
        }
        if (TRAIN && live && ok) net_store<kCols>(g.H2 + row * kNetH + c0, v);
    }
    sy[grp * kRows + r] = p;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    ok = __syncthreads_and(ok);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (tid < kRows && !ok) {
        if (live && g.y) g.y[row] = nanf("");
    } else if (tid < kRows) {   // threads 0 .. kRows - 1: tile row tid (grp 0 of the first quadrants)
        float y = sy[tid];
#pragma unroll
        for (int i = 1; i < 2 * D; ++i) y += sy[i * kRows + tid];
        y += g.b3[0];
        if (live && g.y) g.y[row] = y;
        if (TRAIN) {        // loss = mean((y - t)^2), dy = 2 (y - t) / B
            const float d = live ? y - g.target[row] : 0.0f;
            const float dy = 2.0f * d / (float)g.B;
            sdy[tid] = dy;
            if (live) g.dY[row] = dy;
            float l = d * d / (float)g.B;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
            if (lane == 0) atomicAdd(g.loss, l);
        }
    }
    if (TRAIN) {
        __syncthreads();
        const float dy = sdy[r];
        // ---- dZ2 = dy w3 GELU'(Z2), and dH1 = dZ2 W2 over Z1's accumulator columns
        if (tid == 0) ok = ok && mma_wait(b_w2, 1, g.wait);
        for (int q = kNetChunks; q < 2 * kNetChunks; ++q) {
            float v[kCols];
            const int c0 = (q - kNetChunks) * kNetChunk + grp * kCols;
            net_ld<kCols>(tlane + (uint32_t)(kNetH + c0), v);
#pragma unroll
            for (int e = 0; e < kCols; ++e) v[e] = (dy * sw3[c0 + e]) * gelu_grad(v[e] + sb2[c0 + e]);
            if (live && ok) net_store<kCols>(g.dZ2 + row * kNetH + c0, v);
            chunk(q, kNetChunks, tmem, v);
        }
        ok = ok && mma_wait(b_ch, (uint32_t)((2 * kNetChunks - 1) & 1), g.wait);
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int q = 0; q < kNetChunks; ++q) {   // dZ1 = dH1 GELU'(Z1), Z1 as this thread wrote it above
            float v[kCols];
            const int c0 = q * kNetChunk + grp * kCols;
            net_ld<kCols>(tlane + (uint32_t)c0, v);
            if (live && ok) {
                const float4* z1 = reinterpret_cast<const float4*>(g.Z1 + row * kNetH + c0);
#pragma unroll
                for (int e = 0; e < kCols; e += 4) {
                    const float4 a = z1[e / 4];
                    v[e] *= gelu_grad(a.x); v[e + 1] *= gelu_grad(a.y);
                    v[e + 2] *= gelu_grad(a.z); v[e + 3] *= gelu_grad(a.w);
                }
                net_store<kCols>(g.dZ1 + row * kNetH + c0, v);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (TRAIN) ok = __syncthreads_and(ok);
    else __syncthreads();
    if (TRAIN && !ok && tid < kRows && live) g.dY[row] = nanf("");
    if (!ok) {   // a wait was given up on: flag it, and let copies and MMAs in flight land before shared memory and TMEM go
        if (tid == 0) {
            if (g.err) atomicOr(g.err, 1u);
            if (TRAIN) atomicAdd(g.loss, nanf(""));
            net_drain(b_w1, 0u);
            net_drain(b_w2, w2t ? 1u : 0u);
            if (l1) net_drain(b_l1, 0u);
            if (n_ch) net_drain(b_ch, (uint32_t)((n_ch - 1) & 1));
        }
        __syncthreads();
    }
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"((uint32_t)kNetTmemCols)
                     : "memory");
    }
}

// ------------------------------------------------------------ weight gradients
// dW2 = dZ2^T H1, dW1 = dZ1^T X on the tensor cores (both operands three BF16 terms), db2, db1 and
// dW3 as column sums, over the rows of one split; blockIdx.x = half of the output rows (128 of
// 256), blockIdx.y = split.  A thread owns one column of each operand: its loads are coalesced
// across the warp, eight rows make one 16-byte row of a core matrix, and the column sums fall out
// of the same loads.  Partial sums are added to the zeroed gradient.
constexpr int kGradStage = 64;                                       // rows staged at once
constexpr int kGradA = 128 * kGradStage * 2;                         // one term of dZ2^T (or dZ1^T)
constexpr int kGradB = kNetH * kGradStage * 2;                       // one term of H1^T
constexpr int kGradX = kNetMaxIn * kGradStage * 2;                   // one term of X^T (rows padded)
constexpr int kGradOffA1 = 3 * kGradA;
constexpr int kGradOffB = 2 * 3 * kGradA;
constexpr int kGradOffX = kGradOffB + 3 * kGradB;
constexpr int kGradSmem = kGradOffX + 3 * kGradX;
static_assert(kGradSmem <= 227 * 1024, "shared memory of one CTA");

struct GradArgs {
    int in, kx;
    int64_t B, rows_per_split;
    const float *x, *H1, *H2, *dZ2, *dZ1, *dY;
    float *gW1, *gb1, *gW2, *gb2, *gW3, *gb3;
    float* loss;
    unsigned* err;
    uint32_t wait;
};

__global__ void __launch_bounds__(kNetThreads, 1) k_net_grad(GradArgs g)
{
    extern __shared__ __align__(1024) unsigned char gsm[];
    __shared__ __align__(8) unsigned long long bar;
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int oc = tid & 127, og = tid >> 7;              // output column of the half, row-group half
    const int o = blockIdx.x * 128 + oc;
    const int64_t r_begin = (int64_t)blockIdx.y * g.rows_per_split;
    const int64_t r_end = r_begin + g.rows_per_split < g.B ? r_begin + g.rows_per_split : g.B;
    const uint32_t mb = smem_addr(&bar);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_addr(&tmem_base)), "r"((uint32_t)kNetTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(mb) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;
    float s_b2 = 0.0f, s_b1 = 0.0f, s_w3 = 0.0f, s_b3 = 0.0f;
    bool ok = true;
    int st = 0, n_st = 0;   // stages; thread 0: those whose MMAs were issued
    for (int64_t r0 = r_begin; r0 < r_end; r0 += kGradStage, ++st) {
        if (st > 0) ok = ok && mma_wait(mb, (uint32_t)((st - 1) & 1), g.wait);   // the operands are free again
        // H1^T: thread = column i, eight row groups
#pragma unroll 4
        for (int c = 0; c < kGradStage / 8; ++c) {
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int64_t row = r0 + c * 8 + e;
                v[e] = row < r_end ? __ldg(g.H1 + row * kNetH + tid) : 0.0f;
            }
            net_split8(v, gsm + kGradOffB + (c * (kNetH / 8) + (tid >> 3)) * 128 + (tid & 7) * 16, kGradB);
        }
        // dZ2^T, dZ1^T: thread = output column, half of the row groups; column sums
#pragma unroll 4
        for (int cc = 0; cc < kGradStage / 16; ++cc) {
            const int c = og * (kGradStage / 16) + cc;
            float v[8], u[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int64_t row = r0 + c * 8 + e;
                const bool in_range = row < r_end;
                v[e] = in_range ? __ldg(g.dZ2 + row * kNetH + o) : 0.0f;
                u[e] = in_range ? __ldg(g.dZ1 + row * kNetH + o) : 0.0f;
                s_b2 += v[e];
                s_b1 += u[e];
                if (in_range) {
                    const float dy = __ldg(g.dY + row);
                    s_w3 = fmaf(dy, __ldg(g.H2 + row * kNetH + o), s_w3);
                    s_b3 += dy;
                }
            }
            const int at = (c * 16 + (oc >> 3)) * 128 + (oc & 7) * 16;
            net_split8(v, gsm + at, kGradA);
            net_split8(u, gsm + kGradOffA1 + at, kGradA);
        }
        // X^T: thread = (input f, row group), f padded with zeros
        for (int q = tid; q < g.kx * (kGradStage / 8); q += kNetThreads) {
            const int f = q % g.kx, c = q / g.kx;
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int64_t row = r0 + c * 8 + e;
                v[e] = (row < r_end && f < g.in) ? __ldg(g.x + row * g.in + f) : 0.0f;
            }
            net_split8(v, gsm + kGradOffX + (c * (g.kx / 8) + (f >> 3)) * 128 + (f & 7) * 16, kGradX);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0 && ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int s = 0; s < kGradStage / 16; ++s)
                for (int i = 0; i < 3; ++i)
                    for (int j = 0; i + j < 3; ++j) {   // products above 2^-24
                        const bool acc = st > 0 || s + i + j > 0;
                        net_mma(tmem, net_desc(smem_addr(gsm + i * kGradA + s * 2 * 16 * 128), 16 * 128, 128),
                                net_desc(smem_addr(gsm + kGradOffB + j * kGradB + s * 2 * (kNetH / 8) * 128),
                                         (kNetH / 8) * 128, 128), mma_idesc(kNetH), acc);
                        net_mma(tmem + kNetH, net_desc(smem_addr(gsm + kGradOffA1 + i * kGradA + s * 2 * 16 * 128), 16 * 128, 128),
                                net_desc(smem_addr(gsm + kGradOffX + j * kGradX + s * 2 * (g.kx / 8) * 128),
                                         (uint32_t)(g.kx / 8) * 128, 128), mma_idesc(g.kx), acc);
                    }
            net_commit(mb);
            ++n_st;
        }
    }
    if (st > 0) ok = ok && mma_wait(mb, (uint32_t)((st - 1) & 1), g.wait);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok && lane == 0) {   // a wait was given up on: the warp adds nothing, the loss says so
        atomicOr(g.err, 1u);
        atomicAdd(g.loss, nanf(""));
    }
    if (!ok && tid == 0 && n_st) net_drain(mb, (uint32_t)((n_st - 1) & 1));   // MMAs in flight end before TMEM goes
    if (st > 0 && ok) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // thread: output row 128 x + 32 (w % 4) + lane, 128 of the 256 columns
        const int m = blockIdx.x * 128 + (warp & 3) * 32 + lane;
        const uint32_t tl = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const int half = warp >> 2;
        float v[16];
        for (int c = 0; c < kNetH / 2; c += 16) {
            const int c0 = half * (kNetH / 2) + c;
            net_ld16(tl + (uint32_t)c0, v);
            float4* dst = reinterpret_cast<float4*>(g.gW2 + (int64_t)m * kNetH + c0);
#pragma unroll
            for (int e = 0; e < 4; ++e) atomicAdd(dst + e, make_float4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]));
        }
        if (half * 16 < g.kx) {
            net_ld16(tl + (uint32_t)(kNetH + half * 16), v);
#pragma unroll
            for (int e = 0; e < 16; ++e)
                if (half * 16 + e < g.in) atomicAdd(g.gW1 + (int64_t)m * g.in + half * 16 + e, v[e]);
        }
        atomicAdd(g.gb2 + o, s_b2);
        atomicAdd(g.gb1 + o, s_b1);
        atomicAdd(g.gW3 + o, s_w3);
        if (blockIdx.x == 0 && oc == 0) atomicAdd(g.gb3, s_b3);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"((uint32_t)kNetTmemCols)
                     : "memory");
    }
}

// Weight p of the flat order into the operand images (in inputs, hidden = 256) and W3 behind them.
constexpr int kNetImgW3 = 2 * kNetImgW2 + kNetH * kNetMaxIn;        // elements: W2, W2^T, W1
constexpr int kNetImg = kNetImgW3 + kNetH;

__device__ __forceinline__ void net_write_img(int64_t p, int in, int kx, __nv_bfloat16 w, __nv_bfloat16* img)
{
    const int64_t o2 = (int64_t)kNetH * in + kNetH, o3 = o2 + kNetImgW2 + kNetH;
    if (p >= o3 && p < o3 + kNetH) img[kNetImgW3 + (p - o3)] = w;
    if (p < (int64_t)kNetH * in) {
        img[2 * kNetImgW2 + net_img(kNetH, (int)(p / in), (int)(p % in))] = w;
    } else if (p >= o2 && p < o2 + kNetImgW2) {
        const int o = (int)((p - o2) / kNetH), i = (int)((p - o2) % kNetH);
        img[net_img(kNetH, o, i)] = w;
        img[kNetImgW2 + net_img(kNetH, i, o)] = w;
    }
}
