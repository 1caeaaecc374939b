// perm.cu — oblivious application of sharded permutations, fused with the
// group reshare (generation: fy.cu).
#include <algorithm>

#include "launch.cuh"

namespace orqcu {

// ---------------------------------------------------------------------------
// Application of one group's local permutation fused with that group's
// reshare, for up to two vectors that use the same permutation (ORQ applies
// the data vector and the permutation vector in turn with the same sharded
// permutation, shuffle.h:687-706). dst[k] = src[idx[k]] (+|^) r_j[k]:
// idx = inverse permutation for local_apply_perm (scatter new[pi[i]] = x[i],
// shuffle.h:113-133), idx = the permutation itself for
// local_apply_inverse_perm (shuffle.h:250-270).
//   MODE 0: store both results
//   MODE 2: open the second vector into sigma and scatter the first by it
//           (local_apply_perm of the opened permutation, shuffle.h:702-705)
//   MODE 3: open the first vector into sigma (no stores)
struct ApplyArgs {
    const void* src1[3];
    void* dst1[3];
    const void* src2[3];
    void* dst2[3];
    const int32_t* idx;
    StreamArg g1, g2;
    unsigned long long ch1, ch2;
    unsigned long long n;
    int32_t* sigma;
    int* err;
};

template <int W>
__device__ __forceinline__ void gather_elem(const void* src, int32_t k, uint8_t* dst) {
    if constexpr (W == 4) {
        *reinterpret_cast<uint32_t*>(dst) = __ldg(reinterpret_cast<const uint32_t*>(src) + k);
    } else if constexpr (W == 8) {
        *reinterpret_cast<uint2*>(dst) = __ldg(reinterpret_cast<const uint2*>(src) + k);
    } else {
        *reinterpret_cast<uint4*>(dst) = __ldg(reinterpret_cast<const uint4*>(src) + k);
    }
}
template <int W>
__device__ __forceinline__ void store_elem(void* dst, int32_t k, const uint8_t* v) {
    if constexpr (W == 4) {
        reinterpret_cast<uint32_t*>(dst)[k] = *reinterpret_cast<const uint32_t*>(v);
    } else if constexpr (W == 8) {
        reinterpret_cast<uint2*>(dst)[k] = *reinterpret_cast<const uint2*>(v);
    } else {
        reinterpret_cast<uint4*>(dst)[k] = *reinterpret_cast<const uint4*>(v);
    }
}

// the three shares of elements id[0..E) of src into E*W/16 16-byte words
// (element e at byte e*W); elements at or past n are left unchanged
template <int W, int E, int B>
__device__ __forceinline__ void gather3(const void* const* src, const int32_t (&id)[E], unsigned long long k0,
                                        unsigned long long n, uint4 (&v)[3][B]) {
#pragma unroll
    for (int j = 0; j < 3; j++)
#pragma unroll
        for (int e = 0; e < E; e++) {
            if (k0 + e >= n) continue;
            if constexpr (W == 16) {
                v[j][e] = __ldg(reinterpret_cast<const uint4*>(src[j]) + id[e]);
            } else if constexpr (W == 8) {
                const uint2 x = __ldg(reinterpret_cast<const uint2*>(src[j]) + id[e]);
                if (e & 1) {
                    v[j][e >> 1].z = x.x;
                    v[j][e >> 1].w = x.y;
                } else {
                    v[j][e >> 1].x = x.x;
                    v[j][e >> 1].y = x.y;
                }
            } else {
                const uint32_t x = __ldg(reinterpret_cast<const uint32_t*>(src[j]) + id[e]);
                switch (e & 3) {
                    case 0: v[j][e >> 2].x = x; break;
                    case 1: v[j][e >> 2].y = x; break;
                    case 2: v[j][e >> 2].z = x; break;
                    default: v[j][e >> 2].w = x; break;
                }
            }
        }
}

template <int E>
__device__ __forceinline__ void load_idx(const int32_t* idx, unsigned long long k0, unsigned long long n,
                                         int32_t (&id)[E]) {
#pragma unroll
    for (int e = 0; e < E; e++) id[e] = (k0 + e < n) ? __ldg(idx + k0 + e) : 0;
}

// Zero-sharing of one 16-byte block of a vector: the keystreams of block blk in
// the group stream (r0) and at nonce offset ch (r1), r2 = -(r0 + r1) or
// r0 ^ r1, added to the three shares held at v[.][0]; then v[.][0..B) rotate
// left by one so the next block sits at index 0 (after B calls the order is
// restored). Called from loops kept rolled: two AES bodies per vector instead
// of two per block keep the kernel's loop inside the instruction cache (fully
// unrolled, ten AES-256 bodies stalled every warp on instruction fetch).
template <int W, bool A, int B>
__device__ __forceinline__ void reshare_block(const AesSmem& S, const StreamArg& gs, unsigned long long ch,
                                              unsigned long long blk, uint4 (&v)[3][B]) {
    uint4 r0 = make_uint4(0, 0, 0, 0), r1 = r0;
#pragma unroll 1
    for (int c = 0; c < 2; c++) {  // (rolled: one AES body)
        r0 = r1;
        r1 = keystream_block_n(S, gs.rk, gs.nonce + c * ch, blk);
    }
    uint4 r2;
    if constexpr (A) r2 = Ring<W>::sub(Ring<W>::sub(make_uint4(0, 0, 0, 0), r0), r1);
    else r2 = r0 ^ r1;
    v[0][0] = Share<W, A>::plus(v[0][0], r0);
    v[1][0] = Share<W, A>::plus(v[1][0], r1);
    v[2][0] = Share<W, A>::plus(v[2][0], r2);
    if constexpr (B > 1) {
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const uint4 x = v[j][0];
#pragma unroll
            for (int b = 0; b + 1 < B; b++) v[j][b] = v[j][b + 1];
            v[j][B - 1] = x;
        }
    }
}

// E elements per thread and unit; E*W1 and E*W2 are multiples of 16 bytes.
// Software-pipelined: a unit's gathers are issued in the previous iteration,
// right after that iteration has consumed the same registers, so each random
// gather has a whole iteration of keystream work to arrive in; the next unit's
// indices are loaded at the top of an iteration.
template <int W1, bool A1, int W2, bool A2, int MODE>
__global__ void __launch_bounds__(kAesThreads, 1) k_apply(ApplyArgs a) {
    constexpr int WMIN = (W2 && W2 < W1) ? W2 : W1;
    constexpr int E = 16 / WMIN;
    constexpr int B1 = E * W1 / 16;
    constexpr int B2 = W2 ? E * W2 / 16 : 1;
    extern __shared__ __align__(16) uint32_t sm[];
    aes_stage_tables(sm);
    const AesSmem S(sm);
    const unsigned long long units = ceil_div(a.n, E);
    unsigned long long t = gtid();
    if (t >= units) return;  // no barrier follows the table staging
    const unsigned long long stride = gstride();
    uint4 v1[3][B1], v2[3][B2];
    {
        int32_t id[E];
        load_idx<E>(a.idx, t * E, a.n, id);
        gather3<W1, E, B1>(a.src1, id, t * E, a.n, v1);
        if constexpr (W2 != 0) gather3<W2, E, B2>(a.src2, id, t * E, a.n, v2);
    }
    for (;;) {
        const unsigned long long k0 = t * E;
        const unsigned long long tn = t + stride;
        const bool more = tn < units;
        int32_t idn[E];
        load_idx<E>(a.idx, more ? tn * E : a.n, a.n, idn);
        // ---- vector 2 (the permutation vector in elementwise application)
        uint32_t sig[E];
        if constexpr (W2 != 0) {
#pragma unroll 1
            for (int bb = 0; bb < B2; bb++) reshare_block<W2, A2, B2>(S, a.g2, a.ch2, t * B2 + bb, v2);
            if constexpr (MODE == 0) {
#pragma unroll
                for (int j = 0; j < 3; j++)
#pragma unroll
                    for (int bb = 0; bb < B2; bb++) st16(a.dst2[j], t * B2 + bb, a.n * W2, v2[j][bb]);
            } else if constexpr (MODE == 2) {
                // open (W2 == 4): sigma = sum or xor of the three shares
                uint4 o[B2];
#pragma unroll
                for (int bb = 0; bb < B2; bb++)
                    o[bb] = Share<W2, A2>::plus(Share<W2, A2>::plus(v2[0][bb], v2[1][bb]), v2[2][bb]);
#pragma unroll
                for (int e = 0; e < E; e++) sig[e] = reinterpret_cast<const uint32_t*>(o)[e];
            }
            if (more) gather3<W2, E, B2>(a.src2, idn, tn * E, a.n, v2);
        }
        // ---- vector 1
#pragma unroll 1
        for (int bb = 0; bb < B1; bb++) reshare_block<W1, A1, B1>(S, a.g1, a.ch1, t * B1 + bb, v1);
        if constexpr (MODE == 0) {
#pragma unroll
            for (int j = 0; j < 3; j++)
#pragma unroll
                for (int bb = 0; bb < B1; bb++) st16(a.dst1[j], t * B1 + bb, a.n * W1, v1[j][bb]);
        } else if constexpr (MODE == 2) {
#pragma unroll
            for (int j = 0; j < 3; j++)
#pragma unroll
                for (int e = 0; e < E; e++)
                    if (k0 + e < a.n) {
                        // sigma is an opened permutation; a value outside [0, n)
                        // means corrupted shares: flag it, skip the store
                        if ((unsigned long long)sig[e] < a.n)
                            store_elem<W1>(a.dst1[j], (int32_t)sig[e],
                                           reinterpret_cast<const uint8_t*>(&v1[j][0]) + e * W1);
                        else
                            atomicOr(a.err, 8);
                    }
        } else if constexpr (MODE == 3) {
            uint4 o[B1];
#pragma unroll
            for (int bb = 0; bb < B1; bb++)
                o[bb] = Share<W1, A1>::plus(Share<W1, A1>::plus(v1[0][bb], v1[1][bb]), v1[2][bb]);
#pragma unroll
            for (int e = 0; e < E; e++)
                if (k0 + e < a.n) a.sigma[k0 + e] = reinterpret_cast<const int32_t*>(o)[e];
        }
        if (!more) break;
        gather3<W1, E, B1>(a.src1, idn, tn * E, a.n, v1);
        t = tn;
    }
}

namespace {

template <int W1, bool A1, int W2, bool A2, int MODE>
void launch_apply(Ctx& c, const ApplyArgs& a) {
    constexpr int WMIN = (W2 && W2 < W1) ? W2 : W1;
    constexpr int E = 16 / WMIN;
    auto kern = k_apply<W1, A1, W2, A2, MODE>;
    prep_aes_kernel(kern);
    const unsigned long long units = ceil_div(a.n, E);
    // idx + gathered shares + written shares (the second vector is only read
    // when its result is opened instead of stored)
    const double by = (double)a.n * (4.0 + 6.0 * W1 + (W2 ? (MODE == 0 ? 6.0 : 3.0) * W2 : 0.0));
    const double bl = 2.0 * ((double)ceil_div(a.n * W1, 16) + (W2 ? (double)ceil_div(a.n * W2, 16) : 0.0));
    ProfScope ps(c, "apply_group", by, bl);
    kern<<<aes_grid(c, units), kAesThreads, kAesSmemBytes, c.stream>>>(a);
    ORQ_CUDA_CHECK(cudaGetLastError());
    c.kernels_launched++;
}

// runtime dispatch over the (width, encoding) combinations used by the operators
template <int MODE>
void dispatch_apply(Ctx& c, int w1, bool a1, int w2, bool a2, const ApplyArgs& a) {
#define ORQ_AP(W1v, A1v, W2v, A2v)                                      \
    if (w1 == W1v && a1 == A1v && w2 == W2v && (W2v == 0 || a2 == A2v)) \
        return launch_apply<W1v, A1v, W2v, A2v, MODE>(c, a);
    ORQ_AP(4, false, 0, false)
    ORQ_AP(4, true, 0, false)
    ORQ_AP(8, false, 0, false)
    ORQ_AP(8, true, 0, false)
    ORQ_AP(16, false, 0, false)
    ORQ_AP(16, true, 0, false)
    ORQ_AP(16, false, 4, true)
    ORQ_AP(16, false, 4, false)
    ORQ_AP(8, false, 4, true)
    ORQ_AP(8, true, 4, true)
    ORQ_AP(8, false, 4, false)
    ORQ_AP(8, true, 4, false)
    ORQ_AP(4, true, 4, true)
    ORQ_AP(4, false, 4, true)
    ORQ_AP(4, true, 4, false)
    ORQ_AP(4, false, 4, false)
#undef ORQ_AP
    throw std::invalid_argument("unsupported share width/encoding for permutation application");
}

}  // namespace

// hm_oblivious_apply_sharded_perm / _inverse (shuffle.h:349-412) on one vector.
void op_apply_sharded(Ctx& c, bool arith, int w, size_t n, Sh3 s, ShardedPerm& sp, bool inverse) {
    if (w != 4 && w != 8 && w != 16)
        throw std::invalid_argument("permutation application supports 4, 8 and 16-byte shares");
    const unsigned long long ch = chunks_of((unsigned long long)n * w);
    if (n == 0) return;
    if (inverse) ensure_perm(c, sp);
    Scratch tmp(c, 3 * n * (size_t)w);
    void* other[3] = {tmp.as<uint8_t>(), tmp.as<uint8_t>() + n * (size_t)w,
                      tmp.as<uint8_t>() + 2 * n * (size_t)w};
    void* cur[3] = {s.p[0], s.p[1], s.p[2]};
    for (int step = 0; step < 3; step++) {
        const int g = inverse ? 2 - step : step;
        ApplyArgs a{};
        for (int j = 0; j < 3; j++) {
            a.src1[j] = cur[j];
            a.dst1[j] = other[j];
        }
        a.idx = inverse ? sp.perm[g] : sp.inv[g];
        a.g1 = c.stream_arg(G01 + g);
        a.ch1 = ch;
        a.n = n;
        dispatch_apply<0>(c, w, arith, 0, false, a);
        c.nonce[G01 + g] += 2 * ch;
        for (int j = 0; j < 3; j++) std::swap(cur[j], other[j]);
    }
    // three swaps leave the result in the scratch buffers
    for (int j = 0; j < 3; j++)
        ORQ_CUDA_CHECK(cudaMemcpyAsync(s.p[j], cur[j], n * (size_t)w, cudaMemcpyDeviceToDevice, c.stream));
}

// oblivious_apply_elementwise_perm (shuffle.h:687-706): shuffle x and a copy
// of the permutation with the same sharded permutation, open the shuffled
// permutation and scatter x with it. Three fused kernels, one per group.
void op_apply_elementwise(Ctx& c, bool x_arith, int xw, size_t n, Sh3 x, CSh3 perm) {
    if (n == 0) {
        ShardedPerm sp = next_perm(c, n);
        c.free_perm(sp);
        return;
    }
    ShardedPerm sp = next_perm(c, n);
    const unsigned long long chx = chunks_of((unsigned long long)n * xw);
    const unsigned long long chp = chunks_of((unsigned long long)n * 4);
    Scratch xa(c, 3 * n * (size_t)xw), xb(c, 3 * n * (size_t)xw), pa(c, 3 * n * 4), pb(c, 3 * n * 4);
    void* X[2][3];
    void* Pp[2][3];
    for (int j = 0; j < 3; j++) {
        X[0][j] = xa.as<uint8_t>() + j * n * (size_t)xw;
        X[1][j] = xb.as<uint8_t>() + j * n * (size_t)xw;
        Pp[0][j] = pa.as<uint8_t>() + j * n * 4;
        Pp[1][j] = pb.as<uint8_t>() + j * n * 4;
    }
    for (int g = 0; g < 3; g++) {
        ApplyArgs a{};
        for (int j = 0; j < 3; j++) {
            a.src1[j] = g == 0 ? x.p[j] : X[(g - 1) & 1][j];
            a.dst1[j] = g == 2 ? x.p[j] : X[g & 1][j];
            a.src2[j] = g == 0 ? perm.p[j] : Pp[(g - 1) & 1][j];
            a.dst2[j] = Pp[g & 1][j];
        }
        a.idx = sp.inv[g];
        a.err = c.d_err;
        // per group stream: the x reshare first, then the permutation's
        a.g1 = c.stream_arg(G01 + g);
        a.g2 = c.stream_arg(G01 + g, 2 * chx);
        a.ch1 = chx;
        a.ch2 = chp;
        a.n = n;
        if (g < 2) dispatch_apply<0>(c, xw, x_arith, 4, true, a);
        else dispatch_apply<2>(c, xw, x_arith, 4, true, a);
        c.nonce[G01 + g] += 2 * chx + 2 * chp;
    }
    c.free_perm(sp);
}

// shuffle (shuffle.h:752-757)
void op_shuffle(Ctx& c, bool arith, int w, size_t n, Sh3 s) {
    ShardedPerm sp = next_perm(c, n);
    op_apply_sharded(c, arith, w, n, s, sp, false);
    c.free_perm(sp);
}

// local_apply_perm with a public permutation: dst[sigma[i]] = src[i]
template <int W>
__global__ void k_scatter(CSh3 src, Sh3 dst, const int32_t* sigma, unsigned long long n, int* err) {
    for (unsigned long long i = gtid(); i < n; i += gstride()) {
        const int32_t d = __ldg(sigma + i);
        if ((unsigned long long)(uint32_t)d >= n) {
            atomicOr(err, 8);
            continue;
        }
#pragma unroll
        for (int j = 0; j < 3; j++) {
            uint8_t v[W];
            gather_elem<W>(src.p[j], (int32_t)i, v);
            store_elem<W>(dst.p[j], d, v);
        }
    }
}
void op_scatter(Ctx& c, int w, size_t n, CSh3 src, Sh3 dst, const int32_t* sigma) {
    if (!n) return;
    const unsigned g = plain_grid(c, n);
    if (w == 4) k_scatter<4><<<g, 256, 0, c.stream>>>(src, dst, sigma, n, c.d_err);
    else if (w == 8) k_scatter<8><<<g, 256, 0, c.stream>>>(src, dst, sigma, n, c.d_err);
    else if (w == 16) k_scatter<16><<<g, 256, 0, c.stream>>>(src, dst, sigma, n, c.d_err);
    else throw std::invalid_argument("scatter supports 4, 8, 16-byte shares");
    ORQ_CUDA_CHECK(cudaGetLastError());
    c.kernels_launched++;
}

}  // namespace orqcu
