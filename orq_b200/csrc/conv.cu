// conv.cu — ASharedVector::a2b (a_shared_vector.h:138-144): the arithmetic
// sharing is redistributed as two boolean sharings (redistribute_shares_b,
// replicated_3pc.h:259-262: party 0 shares S0 + S1, party 2 shares S2) whose
// sum, computed by the boolean ripple-carry adder (operators/circuits.h:35-76),
// is the boolean sharing of the value.
//
// The adder works on bit-packed words: bit i of 8W consecutive elements forms
// one word (pack_from), and each of the 8W-1 carry rounds is one AND over the
// ceil(n / 8W) words, c_i = ((c_{i-1} ^ a_i) & (a ^ b)_i) ^ a_i.
#include <algorithm>
#include <type_traits>

#include "launch.cuh"

namespace orqcu {

namespace {

struct RcaArgs {
    const void* a[3];
    const void* b[3];
    void* sum[3];
    StreamArg pair[3];     // nonces at the first carry round
    unsigned long long n;  // elements
    unsigned long long C;  // nonces per carry round (an AND over the packed words)
    uint32_t* park;        // [warps of the grid][W/2][3][16][32] sums of finished slices
    int carry_in;          // subtraction: the carry starts as all ones (inplace_invert)
};

// The masked-swap transpose of a bit matrix (Warren, Hacker's Delight, 7-3) on
// 16 x 32 bits: reg k holds 16 bits of elements k (low half) and k + 16 (high
// half); afterwards reg b holds bit b of elements 0..31. Its own inverse.
__device__ __forceinline__ void transpose16(uint32_t (&x)[16]) {
    const auto stage = [&](const int j, const uint32_t m) {
#pragma unroll
        for (int k = 0; k < 16; k++)
            if (!(k & j)) {
                const uint32_t t = ((x[k] >> j) ^ x[k + j]) & m;
                x[k + j] ^= t;
                x[k] ^= t << j;
            }
    };
    stage(8, 0x00ff00ffu);
    stage(4, 0x0f0f0f0fu);
    stage(2, 0x33333333u);
    stage(1, 0x55555555u);
}

// A warp takes 1024 elements at a time, a lane 32 consecutive ones: one packed
// word of 32 (half a word of 64), whose bits it holds as 32-bit planes, 16
// bits of the elements (a slice) at a time. The carry is then plain logic on
// three words, and what is left is the keystream: 8 blocks a round and stream
// for the warp, computed 16 rounds at once (lane = round, block). Rows pass
// through shared memory so that global accesses are coalesced at any
// alignment. Bound by the T-table lookups; int32, 2^24 elements: 1.64 ms when a
// ballot packed every bit, 0.63 ms
// now (1024 elements 29.6 and 30.0 us a call, 10000 35.4 and 29.1). The 255
// registers that 8 warps leave do not quite hold a slice: 164 bytes a thread are
// spilled for int32, 112 for int64.
constexpr int kRcaThreads = 256;
constexpr int kRcaRow = 36;  // words of a staged row (32, padded for 16-byte reads)
constexpr int kRcaStage = 32 * kRcaRow, kRcaKs = 16 * 3 * 32;  // words per warp

template <int W>
constexpr size_t rca_smem() {
    return kAesSmemBytes + (size_t)(kRcaThreads / 32) * (kRcaStage + kRcaKs) * 4 + (8 * W - 1) * 3 * 2 * sizeof(CtrPre);
}

template <int W>
__global__ void __launch_bounds__(kRcaThreads, 1) k_rca(RcaArgs a) {
    using T = typename std::conditional<W == 4, uint32_t, uint2>::type;
    constexpr int B = 8 * W, NS = W / 2;
    extern __shared__ __align__(16) uint32_t sm[];
    aes_stage_tables(sm);
    const AesSmem S(sm);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    CtrPre* pre = reinterpret_cast<CtrPre*>(sm + kAesSmemBytes / 4);  // [round][stream][byte 13]
    uint32_t* bufs = sm + kAesSmemBytes / 4 + (B - 1) * 3 * 2 * (sizeof(CtrPre) / 4);
    uint32_t* st = bufs + w * (kRcaStage + kRcaKs);
    uint32_t* ks = st + kRcaStage;  // [round of the slice][stream][word]
    uint32_t* park = a.park + ((size_t)blockIdx.x * (kRcaThreads / 32) + w) * (NS * 3 * 16 * 32) + lane;
    const unsigned long long tiles = ceil_div(a.n, 1024);
    const unsigned long long t0 = tiles * blockIdx.x / gridDim.x, t1 = tiles * (blockIdx.x + 1) / gridDim.x;
    // a CTA with one tile (a small call) computes its keystream with every warp,
    // slice s into warp s's buffer, before warp 0 runs the rounds
    const bool shared_ks = t1 - t0 == 1;
    // rounds 16 s + 4 g .. + 3 of the tile whose blocks start at blk
    const auto fill = [&](uint32_t* out, int s, int g, uint32_t blk) {
        const int r = 4 * g + (lane >> 3);
        const int round = min(16 * s + r, B - 2);  // the top bit has no carry out
#pragma unroll 1
        for (int q = 0; q < 3; q++)  // (rolled: one AES body)
            *reinterpret_cast<uint4*>(out + (r * 3 + q) * 32 + 4 * (lane & 7)) =
                keystream_block_pre(S, a.pair[q].rk, pre + (round * 3 + q) * 2, 0, blk + (lane & 7));
    };
    // word wd of this warp's elements of one array, coalesced. Elements past n
    // repeat the last one: their sums are not stored, and no element's sum
    // depends on another.
    const auto fetch = [&](const void* x, unsigned long long e0, int wd, uint32_t (&v)[32]) {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(x) + wd;
#pragma unroll
        for (int i = 0; i < 32; i++) {
            const unsigned long long e = e0 + 32 * i + lane;
            v[i] = __ldg(src + (e < a.n ? e : a.n - 1) * (W / 4));
        }
    };
    // half hf of the fetched words, the lane's own 32 elements packed for transpose16
    const auto rows = [&](const uint32_t (&v)[32], int hf, uint32_t (&r)[16]) {
        __syncwarp();  // the rows before have been read
#pragma unroll
        for (int i = 0; i < 32; i++) st[i * kRcaRow + lane] = v[i];
        __syncwarp();
        const uint4* row = reinterpret_cast<const uint4*>(st + lane * kRcaRow);
        const uint32_t sel = hf ? 0x7632u : 0x5410u;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint4 lo = row[i], hi = row[i + 4];
            r[4 * i + 0] = __byte_perm(lo.x, hi.x, sel);
            r[4 * i + 1] = __byte_perm(lo.y, hi.y, sel);
            r[4 * i + 2] = __byte_perm(lo.z, hi.z, sel);
            r[4 * i + 3] = __byte_perm(lo.w, hi.w, sel);
        }
    };
    for (unsigned long long s0 = t0; s0 < t1;) {
        // tiles of one chunk (65536 blocks a round and stream, 8 a tile)
        const unsigned long long chunk = s0 >> 13, s1 = min(t1, (chunk + 1) << 13);
        __syncthreads();
        for (int i = threadIdx.x; i < (B - 1) * 6; i += kRcaThreads) {
            const int b13 = i & 1, q = (i >> 1) % 3, round = i / 6;
            pre[i] = ctr_pre(S, a.pair[q].rk, a.pair[q].nonce + (unsigned long long)round * a.C + chunk, (uint32_t)b13);
        }
        __syncthreads();
        if (shared_ks) {
#pragma unroll 1
            for (int i = w; i < 4 * NS; i += kRcaThreads / 32)
                fill(bufs + (i >> 2) * (kRcaStage + kRcaKs) + kRcaStage, i >> 2, i & 3, (uint32_t)(s0 & 8191) * 8);
            __syncthreads();
        }
        for (unsigned long long t = s0 + w; t < s1; t += kRcaThreads / 32) {
            const unsigned long long e0 = t * 1024;
            uint32_t c[3];
            c[0] = c[1] = c[2] = a.carry_in ? 0xffffffffu : 0u;
#pragma unroll 1
            for (int s = 0; s < NS; s++) {
                __syncwarp();
                if (!shared_ks) {
#pragma unroll 1
                    for (int g = 0; g < 4; g++) fill(ks, s, g, (uint32_t)(t & 8191) * 8);
                    __syncwarp();
                }
                const uint32_t* kr = shared_ks ? bufs + s * (kRcaStage + kRcaKs) + kRcaStage : ks;
                uint32_t x[3][16], ab[3][16];
#pragma unroll
                for (int p = 0; p < 3; p++) {
                    uint32_t v[32], y[32];  // both in flight at once
                    fetch(a.a[p], e0, s >> 1, v);
                    fetch(a.b[p], e0, s >> 1, y);
                    rows(v, s & 1, x[p]);
                    rows(y, s & 1, ab[p]);
#pragma unroll
                    for (int r = 0; r < 16; r++) ab[p][r] ^= x[p][r];
                    transpose16(x[p]);
                    transpose16(ab[p]);
                }
#pragma unroll
                for (int r = 0; r < 16; r++) {
                    uint32_t K[3], u[3], z[3];
#pragma unroll
                    for (int q = 0; q < 3; q++) K[q] = kr[(r * 3 + q) * 32 + lane];
#pragma unroll
                    for (int p = 0; p < 3; p++) u[p] = c[p] ^ x[p][r];
#pragma unroll
                    for (int p = 0; p < 3; p++) {
                        const int q = (p + 1) % 3, pm = (p + 2) % 3;
                        z[p] = (K[pm] ^ K[p]) ^ (u[p] & ab[p][r]) ^ (u[p] & ab[q][r]) ^ (u[q] & ab[p][r]);
                    }
#pragma unroll
                    for (int p = 0; p < 3; p++) {
                        ab[p][r] ^= c[p];  // the sum bit
                        c[p] = z[p] ^ x[p][r];
                    }
                }
#pragma unroll
                for (int p = 0; p < 3; p++) {
                    transpose16(ab[p]);
#pragma unroll
                    for (int r = 0; r < 16; r++) park[((s * 3 + p) * 16 + r) * 32] = ab[p][r];
                }
            }
            // a share's finished elements, through the staged rows (int64: the
            // high words through the keystream's buffer)
#pragma unroll 1
            for (int p = 0; p < 3; p++) {
#pragma unroll
                for (int wd = 0; wd < W / 4; wd++) {
                    uint32_t lo[16], hi[16];
#pragma unroll
                    for (int r = 0; r < 16; r++) {
                        lo[r] = park[((2 * wd * 3 + p) * 16 + r) * 32];
                        hi[r] = park[(((2 * wd + 1) * 3 + p) * 16 + r) * 32];
                    }
                    __syncwarp();  // the rows before have been stored
                    uint4* row = reinterpret_cast<uint4*>((wd ? ks : st) + lane * kRcaRow);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        row[i] = make_uint4(__byte_perm(lo[4 * i], hi[4 * i], 0x5410), __byte_perm(lo[4 * i + 1], hi[4 * i + 1], 0x5410),
                                            __byte_perm(lo[4 * i + 2], hi[4 * i + 2], 0x5410), __byte_perm(lo[4 * i + 3], hi[4 * i + 3], 0x5410));
                        row[i + 4] = make_uint4(__byte_perm(lo[4 * i], hi[4 * i], 0x7632), __byte_perm(lo[4 * i + 1], hi[4 * i + 1], 0x7632),
                                                __byte_perm(lo[4 * i + 2], hi[4 * i + 2], 0x7632), __byte_perm(lo[4 * i + 3], hi[4 * i + 3], 0x7632));
                    }
                }
                __syncwarp();
#pragma unroll 8
                for (int i = 0; i < 32; i++) {
                    const unsigned long long e = e0 + 32 * i + lane;
                    if (e < a.n) {
                        if constexpr (W == 4) reinterpret_cast<T*>(a.sum[p])[e] = st[i * kRcaRow + lane];
                        else reinterpret_cast<T*>(a.sum[p])[e] = make_uint2(st[i * kRcaRow + lane], ks[i * kRcaRow + lane]);
                    }
                }
            }
        }
        s0 = s1;
    }
}

// S0 + S1 (party 0's local value x(0) + x(1)) mod 2^(8W)
template <typename T>
__global__ void k_add01(CSh3 x, T* out, unsigned long long n) {
    for (unsigned long long i = gtid(); i < n; i += gstride())
        out[i] = reinterpret_cast<const T*>(x.p[0])[i] + reinterpret_cast<const T*>(x.p[1])[i];
}

}  // namespace

// ripple_carry_adder (operators/circuits.h:35-76) of two boolean sharings
void op_rca(Ctx& c, int w, size_t n, CSh3 A, CSh3 Bv, Sh3 sum, bool carry_in) {
    if (w != 4 && w != 8) throw std::invalid_argument("the boolean adder supports 4 and 8-byte shares");
    const unsigned long long B = 8ull * w, cw = (n + B - 1) / B;
    RcaArgs a;
    for (int j = 0; j < 3; j++) {
        a.a[j] = A.p[j];
        a.b[j] = Bv.p[j];
        a.sum[j] = sum.p[j];
        a.pair[j] = c.stream_arg(PAIR0 + j);
    }
    a.n = n;
    a.C = chunks_of(cw * (unsigned long long)w);
    a.carry_in = carry_in;
    if (n) {
        // CTAs of 8 warps; small calls spread over the SMs, a tile each
        const unsigned grid = (unsigned)std::min<unsigned long long>(ceil_div(n, 1024), (unsigned long long)c.num_sms);
        Scratch park(c, (size_t)grid * (kRcaThreads / 32) * (w / 2) * 3 * 16 * 32 * 4);
        a.park = park.as<uint32_t>();
        const auto kern = w == 4 ? &k_rca<4> : &k_rca<8>;
        const size_t smem = w == 4 ? rca_smem<4>() : rca_smem<8>();
        ORQ_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        ProfScope ps(c, "boolean_adder", 9.0 * w * n, 3.0 * (double)(B - 1) * (double)ceil_div(cw * w, 16));
        kern<<<grid, kRcaThreads, smem, c.stream>>>(a);
        ORQ_CUDA_CHECK(cudaGetLastError());
        c.kernels_launched++;
    }
    for (int q = 0; q < 3; q++) c.nonce[PAIR0 + q] += (B - 1) * a.C;
}

// BSharedVector::operator- (b_shared_vector.h:620-622): a + ~b + 1
void op_sub_b(Ctx& c, int w, size_t n, CSh3 x, CSh3 y, Sh3 z) {
    const size_t n1 = std::max<size_t>(n, 1);
    Scratch nb(c, 3 * n1 * w);
    Sh3 NY;
    for (int j = 0; j < 3; j++) NY.p[j] = nb.as<uint8_t>() + j * n1 * w;
    op_not(c, w, n, y, NY);
    op_rca(c, w, n, x, CSh3{{NY.p[0], NY.p[1], NY.p[2]}}, z, true);
}

void op_a2b(Ctx& c, int w, size_t n, CSh3 x, Sh3 y) {
    if (w != 4 && w != 8) throw std::invalid_argument("a2b supports 4 and 8-byte shares");
    const size_t n1 = std::max<size_t>(n, 1);
    Scratch v(c, n1 * w), fb(c, 3 * n1 * w), sb(c, 3 * n1 * w);
    Sh3 F, G;
    for (int j = 0; j < 3; j++) {
        F.p[j] = fb.as<uint8_t>() + j * n1 * w;
        G.p[j] = sb.as<uint8_t>() + j * n1 * w;
    }
    if (n) {
        if (w == 4) k_add01<uint32_t><<<plain_grid(c, n), 256, 0, c.stream>>>(x, v.as<uint32_t>(), n);
        else k_add01<unsigned long long><<<plain_grid(c, n), 256, 0, c.stream>>>(x, v.as<unsigned long long>(), n);
        ORQ_CUDA_CHECK(cudaGetLastError());
        c.kernels_launched++;
    }
    // redistribute_shares_b: party 0 shares x(0) + x(1), then party 2 its x(0)
    op_secret_share(c, false, w, n, v.p, 0, F);
    op_secret_share(c, false, w, n, x.p[2], 2, G);
    op_rca(c, w, n, CSh3{{F.p[0], F.p[1], F.p[2]}}, CSh3{{G.p[0], G.p[1], G.p[2]}}, y, false);
}

}  // namespace orqcu
