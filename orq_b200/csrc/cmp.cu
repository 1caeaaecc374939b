// cmp.cu — the compare circuit and the bitonic sorting network.
//
// BSharedVector::_compare (include/core/operators/circuits.h:231-295) with
// bit_same (containers/b_shared_vector.h:164-178): log2(8W) AND rounds of a
// prefix-AND over ~(x^y), one AND for ((eq>>1)^eq) & x, a local parity, and a
// sign fix-up on bits packed 8W per word with one more AND (the OR of
// operator|=, b_shared_vector.h:450-455). bitonic_sort
// (operators/sorting.h:266-353) runs one compare per pair and stage followed
// by two multiplexes (operators/common.h:20-28).
//
// In loopback every AND round of a pair is local to the thread that holds the
// pair, so a whole compare or network stage is one kernel and the circuit runs
// in registers.
#include <algorithm>
#include <cstring>
#include <memory>
#include <string>
#include <type_traits>
#include <vector>

#include "launch.cuh"

namespace orqcu {

namespace {

// Threads (= pairs) per CTA of k_rows_cmp. The AES tables take 128 KiB of shared
// memory, so one CTA runs per SM; the per-warp keystream buffers take the rest
// (3 KiB per warp for int32, 6.75 KiB for int64).
template <int W>
constexpr int cmp_threads() { return W == 4 ? 512 : 448; }

// bit_same rounds: log2 of the share's bit width
template <int W>
constexpr int cmp_levels() { return W == 4 ? 5 : (W == 8 ? 6 : 7); }

template <typename T>
struct CmpArgs {
    const T* key[3];    // quicksort: the rows
    const T* x[3];      // compare: this
    const T* y[3];      // compare: other
    T* eq[3];
    T* gt[3];
    StreamArg pair[3];  // nonces at the start of the compare
    unsigned long long C, Cp;  // nonces per full-size and per packed AND call
    unsigned long long m;      // pairs
    // quicksort's compare: with q = idx[p], pair p is (key[ord[q]],
    // key[ord[head[q]]]), and only the opened gt bit is kept, at cb[q]
    const uint32_t* ord;
    const uint32_t* idx;
    const int32_t* head;
    uint8_t* cb;
};

template <typename T>
__device__ __forceinline__ T ashr(T v, int s) {
    if constexpr (sizeof(T) == 16) return (T)((__int128)v >> s);
    else return (T)((typename std::make_signed<T>::type)v >> s);
}

// parity of the bits of v
template <typename T>
__device__ __forceinline__ int parity(T v) {
    if constexpr (sizeof(T) == 16) return (__popcll((unsigned long long)v) ^ __popcll((unsigned long long)(v >> 64))) & 1;
    else return __popcll((unsigned long long)v) & 1;
}

// binary and_b of one element for all three parties: z_p = r_p ^ x_p&y_p ^
// x_p&y_{p+1} ^ x_{p+1}&y_p, r_p = K[p-1] ^ K[p]
template <typename T>
__device__ __forceinline__ void and3(const T x[3], const T y[3], const T k[3], T z[3]) {
    const T r[3] = {(T)(k[2] ^ k[0]), (T)(k[0] ^ k[1]), (T)(k[1] ^ k[2])};
#pragma unroll
    for (int p = 0; p < 3; p++) {
        const int q = (p + 1) % 3;
        z[p] = r[p] ^ (x[p] & y[p]) ^ (x[p] & y[q]) ^ (x[q] & y[p]);
    }
}

// bit_same (b_shared_vector.h:164-178) of one pair for all parties: the
// prefix-AND of ~(a ^ b) from the MSB down; AND round lev uses keystream call
// lev (kword(call, stream) is this thread's word of that call).
template <typename T, typename KW>
__device__ __forceinline__ void bit_same3(const T (&A)[3], const T (&Bv)[3], const KW& kword, T (&Sm)[3]) {
    constexpr int L = cmp_levels<sizeof(T)>();
#pragma unroll
    for (int j = 0; j < 3; j++) Sm[j] = ~(A[j] ^ Bv[j]);
#pragma unroll
    for (int lev = 0; lev < L; lev++) {
        T Tm[3], K[3], Z[3];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            Tm[j] = ashr(Sm[j], 1 << lev);
            K[j] = kword(lev, j);
        }
        and3(Sm, Tm, K, Z);
#pragma unroll
        for (int j = 0; j < 3; j++) Sm[j] = Z[j];
    }
}

// The rest of _compare (circuits.h:249-292) once bit_same is in Sm: gt =
// parity(((eq >> 1) ^ eq) & this) on keystream call L, then the signed fix-up
// on words of 8W packed pairs with one packed AND whose keystream block is kp
// (this warp's [stream][word]). A warp holds pairs [p0w, p0w + 32); for 8-byte
// shares two warps make one packed word, exchanged through `ballots` (all of
// a word's warps must call this). Returns the masked gt bit of the pair.
template <typename T, typename KW>
__device__ __forceinline__ void gt_bits3(const T (&A)[3], const T (&Bv)[3], const T (&Sm)[3], bool valid,
                                         unsigned long long p, unsigned long long p0w, int warp,
                                         const KW& kword, const uint32_t (*kp)[4],
                                         uint32_t (*ballots)[3][3], T (&gt)[3]) {
    constexpr int W = sizeof(T);
    constexpr int B = 8 * W;
    constexpr int L = cmp_levels<W>();
    T G[3];
    {
        T Gi[3], K[3];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            Gi[j] = ashr(Sm[j], 1) ^ Sm[j];
            K[j] = kword(L, j);
        }
        and3(Gi, A, K, G);
    }
    uint32_t b1[3], b2[3], br[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
        b1[j] = __ballot_sync(0xffffffffu, valid && ((A[j] >> (B - 1)) & 1));
        b2[j] = __ballot_sync(0xffffffffu, valid && ((Bv[j] >> (B - 1)) & 1));
        br[j] = __ballot_sync(0xffffffffu, valid && parity(G[j]));
    }
    T s1[3], s2[3], r[3];
    if constexpr (W == 4) {
#pragma unroll
        for (int j = 0; j < 3; j++) {
            s1[j] = b1[j];
            s2[j] = b2[j];
            r[j] = br[j];
        }
    } else {
        // W / 4 warps per packed word of 8W pairs
        constexpr int WPW = W / 4;
        const int lane = threadIdx.x & 31;
        // a barrier of the word's own warps (every warp of the CTA gets here)
        const auto meet = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + warp / WPW), "n"(32 * WPW) : "memory"); };
        meet();
        if (lane == 0)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                ballots[warp][0][j] = b1[j];
                ballots[warp][1][j] = b2[j];
                ballots[warp][2][j] = br[j];
            }
        meet();
        const int w0 = warp & ~(WPW - 1);
#pragma unroll
        for (int j = 0; j < 3; j++) {
            s1[j] = s2[j] = r[j] = 0;
#pragma unroll
            for (int k = 0; k < WPW; k++) {
                s1[j] |= (T)ballots[w0 + k][0][j] << (32 * k);
                s2[j] |= (T)ballots[w0 + k][1][j] << (32 * k);
                r[j] |= (T)ballots[w0 + k][2][j] << (32 * k);
            }
        }
    }
    {
        // r ^= s2 ; s2 ^= s1 ; s2 = ~(~s2 & ~r) ; s1 ^= s2
        T ns2[3], nr[3], K[3], Z[3];
        const unsigned long long c = p0w / B;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const T rr = r[j] ^ s2[j];
            const T ss = s2[j] ^ s1[j];
            ns2[j] = ~ss;
            nr[j] = ~rr;
            if constexpr (W == 4) K[j] = (T)kp[j][c & 3];
            else if constexpr (W == 8) K[j] = (T)kp[j][2 * (c & 1)] | ((T)kp[j][2 * (c & 1) + 1] << 32);
            else K[j] = (T)kp[j][0] | ((T)kp[j][1] << 32) | ((T)kp[j][2] << 64) | ((T)kp[j][3] << 96);
        }
        and3(ns2, nr, K, Z);
#pragma unroll
        for (int j = 0; j < 3; j++) s1[j] ^= ~Z[j];
    }
    const int bitpos = (int)(p % B);
#pragma unroll
    for (int j = 0; j < 3; j++) gt[j] = (s1[j] >> bitpos) & 1;
}

// ---- _compare and operator== of a whole vector --------------------------------
// A lane takes one 16-byte unit of every share, E = 16 / W pairs, so a call's
// keystream is one block a stream that the lane computes itself: nothing is
// staged, no block is computed for padding, and 16 warps run. The packed sign
// fix-up is bitwise, and word c's draw sits in block c W / 16: pair p needs bit
// p % 128 of block p / 128, so the lane works on its own E bits; a warp computes
// the packed blocks of its next 32 passes at once. CTAs take contiguous ranges;
// long ones go chunk by chunk with the constant parts of AES rounds 1 and 2
// (CtrPre). Bound by the T-table lookups. Staged through shared memory (a warp's
// blocks spread over its lanes) and now: 2^24 int32 pairs == 1.81 and 1.47 ms, >
// 2.73 and 1.81 ms; the 56 compares of a quicksort of 2^22 int64 rows 94 and 68 ms.
constexpr int kCmpWarps = kAesThreads / 32;
// A CTA with at most this many passes (a small call) first computes their
// keystream with all its warps: the three blocks of up to eight calls in a row
// took one warp 11 us (> of 1000 int32 pairs: 22.6 and 11.2 us).
constexpr int kCmpSolo = 4;
template <int W, int MODE>
constexpr int cmp_calls() { return cmp_levels<W>() + (MODE == 2 ? 0 : 1); }

template <typename T, int MODE>  // 1: compare, 2: equality, 3: quicksort's compare
__global__ void __launch_bounds__(kAesThreads, 1) k_cmp(CmpArgs<T> a) {
    constexpr int W = sizeof(T), E = 16 / W, L = cmp_levels<W>();
    constexpr int CALLS = cmp_calls<W, MODE>();
    extern __shared__ __align__(16) uint32_t sm[];
    uint4* solo_ks = reinterpret_cast<uint4*>(sm + kAesSmemBytes / 4);  // [pass][call][stream][lane]
    __shared__ CtrPre pre[CALLS][3][2];       // [call][stream][byte 13]
    __shared__ uint4 pk[kCmpWarps][3][32];    // packed blocks of a warp's next passes
    aes_stage_tables(sm);
    const AesSmem S(sm);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // passes: 32 lanes, 32 units each
    const unsigned long long passes = ceil_div(a.m, 32 * E);
    const unsigned long long i0 = passes * blockIdx.x / gridDim.x, i1 = passes * (blockIdx.x + 1) / gridDim.x;
    const bool big = i1 - i0 >= 4 * kCmpWarps, solo = passes <= (unsigned long long)gridDim.x * kCmpSolo;
    if (solo) {
        constexpr int JOBS = (CALLS + (MODE != 2)) * 3;  // per pass; the packed call last
#pragma unroll 1
        for (int i = w; i < (int)(i1 - i0) * JOBS; i += kCmpWarps) {
            const int ps = i / JOBS, call = (i % JOBS) / 3, q = i % 3;
            const unsigned long long it = i0 + ps;
            const bool packed = call == CALLS;
            const uint4 k = keystream_block_n(S, a.pair[q].rk, a.pair[q].nonce + (unsigned long long)(packed ? L + 1 : call) * a.C,
                                              packed ? it * (32 * E) / 128 : it * 32 + lane);
            if (packed) pk[ps][q][0] = k;  // (the same in every lane)
            else solo_ks[((ps * CALLS + call) * 3 + q) * 32 + lane] = k;
        }
        __syncthreads();
    }
    for (unsigned long long s0 = i0; s0 < i1;) {
        const unsigned long long s1 = big ? min(i1, (s0 / 2048 + 1) * 2048) : i1;  // one chunk: 65536 units
        if (big) {
            __syncthreads();
            for (int i = threadIdx.x; i < CALLS * 6; i += kAesThreads) {
                const int q = (i >> 1) % 3, call = i / 6;
                pre[call][q][i & 1] =
                    ctr_pre(S, a.pair[q].rk, a.pair[q].nonce + (unsigned long long)call * a.C + s0 / 2048, (uint32_t)i & 1u);
            }
            __syncthreads();
        }
        for (unsigned long long ib = s0 + w; ib < s1; ib += 32 * kCmpWarps) {
            if (MODE != 2 && !solo) {
                const unsigned long long it = ib + (unsigned long long)lane * kCmpWarps;
                __syncwarp();
                if (it < s1)
#pragma unroll 1
                    for (int q = 0; q < 3; q++)
                        pk[w][q][lane] = keystream_block_n(
                            S, a.pair[q].rk, a.pair[q].nonce + (unsigned long long)(L + 1) * a.C, it * (32 * E) / 128);
                __syncwarp();
            }
            for (int g = 0; g < 32; g++) {
                const unsigned long long it = ib + (unsigned long long)g * kCmpWarps;
                if (it >= s1) break;
                const unsigned long long u = it * 32 + lane, p = u * E;
                T A[E][3], Sm[E][3], G[E][3];
                uint32_t sa[3] = {0, 0, 0}, sb[3] = {0, 0, 0};  // sign bits, bit e = pair p + e
                uint32_t xi[E], xr[E], yr[E];
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    union {
                        uint4 v;
                        T t[E];
                    } x, y;
                    if constexpr (MODE == 3) {
#pragma unroll
                        for (int e = 0; e < E; e++) {
                            x.t[e] = y.t[e] = 0;
                            if (p + e < a.m) {
                                if (j == 0) {
                                    xi[e] = a.idx[p + e];
                                    xr[e] = a.ord[xi[e]];
                                    yr[e] = a.ord[a.head[xi[e]]];
                                }
                                x.t[e] = a.key[j][xr[e]];
                                y.t[e] = a.key[j][yr[e]];
                            }
                        }
                    } else {
                        x.v = ld16(a.x[j], u, a.m * W);
                        y.v = ld16(a.y[j], u, a.m * W);
                    }
#pragma unroll
                    for (int e = 0; e < E; e++) {
                        A[e][j] = x.t[e];
                        Sm[e][j] = ~(x.t[e] ^ y.t[e]);
                        sa[j] |= (uint32_t)(x.t[e] >> (8 * W - 1)) << e;
                        sb[j] |= (uint32_t)(y.t[e] >> (8 * W - 1)) << e;
                    }
                }
                // bit_same's L prefix ANDs, then gt = ((eq >> 1) ^ eq) & this
#pragma unroll 1
                for (int call = 0; call < CALLS; call++) {
                    union {
                        uint4 v;
                        T t[E];
                    } k[3];
                    // the stream loop is rolled: with one AES body the loop stays
                    // inside the instruction cache (three took 1.2 times as long);
                    // each pass appends stream q
                    k[1].v = k[2].v = make_uint4(0, 0, 0, 0);
#pragma unroll 1
                    for (int q = 0; q < 3; q++) {
                        k[0].v = k[1].v;
                        k[1].v = k[2].v;
                        if (solo)
                            k[2].v = solo_ks[((w * CALLS + call) * 3 + q) * 32 + lane];
                        else
                            k[2].v = keystream_block_pre(S, a.pair[q].rk, big ? pre[call][q] : nullptr,
                                                         a.pair[q].nonce + (unsigned long long)call * a.C, u);
                    }
                    const int sh = call < L ? 1 << call : 1;
#pragma unroll
                    for (int e = 0; e < E; e++) {
                        const T K[3] = {k[0].t[e], k[1].t[e], k[2].t[e]};
                        T X[3], Y[3];
#pragma unroll
                        for (int j = 0; j < 3; j++) {
                            const T t = ashr(Sm[e][j], sh);
                            X[j] = call < L ? Sm[e][j] : t ^ Sm[e][j];
                            Y[j] = call < L ? t : A[e][j];
                        }
                        and3(X, Y, K, G[e]);
                        if (call < L)
#pragma unroll
                            for (int j = 0; j < 3; j++) Sm[e][j] = G[e][j];
                    }
                }
                union {
                    uint4 v;
                    T t[E];
                } o;
                if constexpr (MODE != 3) {
#pragma unroll
                    for (int j = 0; j < 3; j++) {
#pragma unroll
                        for (int e = 0; e < E; e++) o.t[e] = Sm[e][j] & 1;
                        st16(a.eq[j], u, a.m * W, o.v);
                    }
                }
                if constexpr (MODE != 2) {
                    // r = parity ^ s2; s2 ^= s1; s2 = ~(~s2 & ~r) (one AND); gt = s1 ^ s2
                    uint32_t ns2[3], nr[3], K[3], Z[3];
#pragma unroll
                    for (int j = 0; j < 3; j++) {
                        uint32_t r = sb[j];
#pragma unroll
                        for (int e = 0; e < E; e++) r ^= (uint32_t)parity(G[e][j]) << e;
                        ns2[j] = ~(sb[j] ^ sa[j]);
                        nr[j] = ~r;
                        const uint32_t bit = (uint32_t)p & 127u;
                        K[j] = reinterpret_cast<const uint32_t*>(&pk[w][j][g])[bit >> 5] >> (bit & 31u);
                    }
                    and3(ns2, nr, K, Z);
                    if constexpr (MODE == 3) {
                        const uint32_t gt = sa[0] ^ sa[1] ^ sa[2] ^ ~(Z[0] ^ Z[1] ^ Z[2]);
#pragma unroll
                        for (int e = 0; e < E; e++)
                            if (p + e < a.m) a.cb[xi[e]] = (uint8_t)((gt >> e) & 1);
                    } else {
#pragma unroll
                        for (int j = 0; j < 3; j++) {
                            const uint32_t gt = sa[j] ^ ~Z[j];
#pragma unroll
                            for (int e = 0; e < E; e++) o.t[e] = (gt >> e) & 1;
                            st16(a.gt[j], u, a.m * W, o.v);
                        }
                    }
                }
            }
        }
        s0 = s1;
    }
}

// ---- compare_rows and swap over several columns -------------------------------
// compare_rows (operators/sorting.h:80-108) runs _compare on every key column,
// in order, and folds key k >= 1 in with two ANDs: gt ^= new_gt & eq, then
// eq &= new_eq. The calls of key k follow each other on the PAIR streams:
// L + 1 full calls and one packed call for the compare, then (k >= 1) the two
// fold calls. A key's keystream is staged per warp exactly as in a compare.
constexpr int kMaxRowKeys = 8;
constexpr int kMaxRowCols = 40;

template <typename T>
struct RowsCmpArgs {
    const T* x[kMaxRowKeys][3];  // bitonic: the key columns (x and y the same)
    const T* y[kMaxRowKeys][3];
    int desc[kMaxRowKeys];
    int nkeys;
    T* gt[3];            // the masked comparison bit per pair
    StreamArg pair[3];   // nonces at the first call
    unsigned long long C, Cp, m;
    int hs;              // bitonic half-box size 2^hs, or -1: pair p is (x[p], y[p])
    int first;
};

// pair p's two rows in a bitonic stage: the box of 2h rows that holds it, row
// k of the first half against row k (or, at j == 0, row h-1-k) of the second
__device__ __forceinline__ void bitonic_rows(unsigned long long p, int hs, int first,
                                             unsigned long long& xi, unsigned long long& yi) {
    const unsigned long long h = 1ull << hs, cb = p >> hs, k = p & (h - 1);
    xi = (cb << (hs + 1)) + k;
    yi = first ? (cb << (hs + 1)) + 2 * h - 1 - k : (cb << (hs + 1)) + h + k;
}

template <typename T>
__global__ void __launch_bounds__(cmp_threads<sizeof(T)>(), 1) k_rows_cmp(RowsCmpArgs<T> a) {
    constexpr int W = sizeof(T);
    constexpr int B = 8 * W;
    constexpr int L = cmp_levels<W>();
    constexpr int NCALL = L + 3;
    constexpr int WORDS = 32 * W / 4;
    constexpr int NB = 32 * W / 16;
    constexpr int kThreads = cmp_threads<W>();
    extern __shared__ __align__(16) uint32_t sm[];
    __shared__ uint32_t ksp[kThreads / 32][3][4];
    __shared__ uint32_t ballots[kThreads / 32][3][3];
    aes_stage_tables(sm);
    const AesSmem S(sm);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t* myks = sm + kAesSmemBytes / 4 + (size_t)warp * NCALL * 3 * WORDS;
    auto kword = [&](int call, int q) -> T {
        const uint32_t* w = myks + (call * 3 + q) * WORDS;
        if constexpr (W == 4) return (T)w[lane];
        else return (T)w[2 * lane] | ((T)w[2 * lane + 1] << 32);
    };
    for (unsigned long long base = (unsigned long long)blockIdx.x * blockDim.x; base < a.m;
         base += (unsigned long long)gridDim.x * blockDim.x) {
        const unsigned long long p0w = base + warp * 32, p = p0w + lane;
        const bool valid = p < a.m;
        unsigned long long xi = p, yi = p;
        if (a.hs >= 0) bitonic_rows(p, a.hs, a.first, xi, yi);
        T G[3] = {0, 0, 0}, E[3] = {0, 0, 0};
        unsigned long long koff = 0;  // nonce offset of key k's first call
        for (int k = 0; k < a.nkeys; k++) {
            T X[3] = {0, 0, 0}, Y[3] = {0, 0, 0};
            if (valid)
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    X[j] = a.x[k][j][xi];
                    Y[j] = a.y[k][j][yi];
                }
            const int ncall = k ? L + 3 : L + 1;
            __syncwarp();  // the previous key's keystream has been read
            for (int idx = lane; idx < ncall * 3 * NB; idx += 32) {
                const int call = idx / (3 * NB), q = (idx / NB) % 3, b = idx % NB;
                const unsigned long long off =
                    koff + (call <= L ? (unsigned long long)call * a.C
                                      : (unsigned long long)(L + 1) * a.C + a.Cp + (unsigned long long)(call - L - 1) * a.C);
                const uint4 ks = keystream_block_n(S, a.pair[q].rk, a.pair[q].nonce + off, p0w * W / 16 + b);
                uint32_t* o = myks + (call * 3 + q) * WORDS + b * 4;
                o[0] = ks.x;
                o[1] = ks.y;
                o[2] = ks.z;
                o[3] = ks.w;
            }
            if (lane < 3) {
                const uint4 ks = keystream_block_n(S, a.pair[lane].rk,
                                                   a.pair[lane].nonce + koff + (unsigned long long)(L + 1) * a.C,
                                                   (p0w / B) * W / 16);
                ksp[warp][lane][0] = ks.x;
                ksp[warp][lane][1] = ks.y;
                ksp[warp][lane][2] = ks.z;
                ksp[warp][lane][3] = ks.w;
            }
            __syncwarp();
            T A[3], Bv[3], Sm[3], g[3];
#pragma unroll
            for (int j = 0; j < 3; j++) {
                A[j] = a.desc[k] ? Y[j] : X[j];
                Bv[j] = a.desc[k] ? X[j] : Y[j];
            }
            bit_same3(A, Bv, kword, Sm);
            gt_bits3(A, Bv, Sm, valid, p, p0w, warp, kword, ksp[warp], ballots, g);
            if (k == 0) {
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    G[j] = g[j];
                    E[j] = Sm[j] & 1;
                }
            } else {
                T K[3], Z[3], e[3];
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    K[j] = kword(L + 1, j);
                    e[j] = Sm[j] & 1;
                }
                and3(g, E, K, Z);
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    G[j] ^= Z[j];
                    K[j] = kword(L + 2, j);
                }
                and3(E, e, K, Z);
#pragma unroll
                for (int j = 0; j < 3; j++) E[j] = Z[j];
            }
            koff += (unsigned long long)ncall * a.C + a.Cp;
        }
        if (valid)
#pragma unroll
            for (int j = 0; j < 3; j++) a.gt[j][p] = G[j] & 1;
    }
}

// swap (operators/sorting.h:146-212) of nbool B-shared then narith A-shared
// column pairs with the same bits: per column tmp = multiplex(b, x, y),
// y = multiplex(b, y, x), x = tmp (operators/common.h:20-49), two AND (or
// multiply_a) calls on the PAIR streams, columns in order. With b2a the
// arithmetic columns use b2a_bit(bits) (replicated_3pc.h:220-251, three
// arithmetic calls after the boolean columns), as bitonic_sort does for its
// A-shared data; otherwise `bits` is already A-shared. One thread owns 16/W
// consecutive pairs and one AES block per stream and call.
template <typename T>
struct RowsSwapArgs {
    T* x[kMaxRowCols][3];
    T* y[kMaxRowCols][3];
    int nbool, narith, b2a;
    const T* bits[3];
    StreamArg pair[3];  // nonces at the first swap call
    unsigned long long C, m;
    int hs, first;      // bitonic mapping as in RowsCmpArgs (hs < 0: none)
};

// keystream of one 16-byte unit u of a call that starts `off` nonces past the
// PAIR streams' nonces: K[e][stream] is element e's word of each stream
template <typename T, int E>
__device__ __forceinline__ void unit_keystream(const AesSmem& S, const StreamArg (&pair)[3],
                                               unsigned long long off, unsigned long long u, T (&K)[E][3]) {
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const uint4 b = keystream_block_n(S, pair[q].rk, pair[q].nonce + off, u);
        if constexpr (sizeof(T) == 4) {
            K[0][q] = b.x;
            K[1][q] = b.y;
            K[2][q] = b.z;
            K[3][q] = b.w;
        } else {
            K[0][q] = (T)b.x | ((T)b.y << 32);
            K[1][q] = (T)b.z | ((T)b.w << 32);
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(kAesThreads, 1) k_rows_swap(RowsSwapArgs<T> a) {
    constexpr int W = sizeof(T);
    constexpr int E = 16 / W;
    extern __shared__ __align__(16) uint32_t sm[];
    aes_stage_tables(sm);
    const AesSmem S(sm);
    const unsigned long long units = ceil_div(a.m, (unsigned long long)E);
    for (unsigned long long u = gtid(); u < units; u += gstride()) {
        auto rows = [&](int e, unsigned long long& xi, unsigned long long& yi) {
            const unsigned long long p = u * E + e;
            xi = yi = p;
            if (a.hs >= 0) bitonic_rows(p, a.hs, a.first, xi, yi);
        };
        auto ok = [&](int e) { return u * E + e < a.m; };
        T bt[E][3];
#pragma unroll
        for (int e = 0; e < E; e++)
#pragma unroll
            for (int j = 0; j < 3; j++) bt[e][j] = ok(e) ? a.bits[j][u * E + e] : (T)0;
        unsigned long long call = 0;
        T K[E][3];
#define ORQ_NEXT_CALL() (unit_keystream(S, a.pair, call++ * a.C, u, K))
#pragma unroll 1
        for (int c = 0; c < a.nbool; c++) {
            T D[E][3];
#pragma unroll
            for (int e = 0; e < E; e++) {
                unsigned long long xi, yi;
                rows(e, xi, yi);
#pragma unroll
                for (int j = 0; j < 3; j++) D[e][j] = ok(e) ? a.x[c][j][xi] ^ a.y[c][j][yi] : (T)0;
            }
            // x' = x ^ (ext(b) & (y ^ x)) on the first call, y' on the second
#pragma unroll 1  // one AES call in flight keeps the tile in registers
            for (int side = 0; side < 2; side++) {
                ORQ_NEXT_CALL();
#pragma unroll
                for (int e = 0; e < E; e++) {
                    if (!ok(e)) continue;
                    unsigned long long xi, yi;
                    rows(e, xi, yi);
                    T Ex[3], Z[3];
#pragma unroll
                    for (int j = 0; j < 3; j++) Ex[j] = (bt[e][j] & 1) ? ~(T)0 : (T)0;  // extend_lsb
                    and3(Ex, D[e], K[e], Z);
#pragma unroll
                    for (int j = 0; j < 3; j++) {
                        T* const v = side ? a.y[c][j] + yi : a.x[c][j] + xi;
                        *v ^= Z[j];
                    }
                }
            }
        }
        if (a.narith == 0) continue;
        if (a.b2a) {
            // b2a_bit: d = s0 - s1 from two zero-sharings, then d * d on the third
            T d[E][3];
#pragma unroll 1  // one AES call in flight keeps the tile in registers
            for (int t = 0; t < 3; t++) {
                ORQ_NEXT_CALL();
#pragma unroll
                for (int e = 0; e < E; e++) {
                    T z[3];
#pragma unroll
                    for (int p = 0; p < 3; p++) z[p] = K[e][(p + 2) % 3] - K[e][p];
                    if (t == 0) {
#pragma unroll
                        for (int p = 0; p < 3; p++) d[e][p] = z[p];
                        d[e][0] += (bt[e][0] ^ bt[e][1]) & 1;  // P0 folds its two masked shares
                    } else if (t == 1) {
#pragma unroll
                        for (int p = 0; p < 3; p++) d[e][p] -= z[p];
                        d[e][1] -= bt[e][2] & 1;  // P1 adds its second masked share to s1
                    } else {
#pragma unroll
                        for (int p = 0; p < 3; p++) {
                            const int q = (p + 1) % 3;
                            bt[e][p] = z[p] + d[e][p] * d[e][p] + d[e][p] * d[e][q] + d[e][q] * d[e][p];
                        }
                    }
                }
            }
        }
        // bt now holds A-shared bits
#pragma unroll 1
        for (int c = a.nbool; c < a.nbool + a.narith; c++) {
            T D[E][3];
#pragma unroll
            for (int e = 0; e < E; e++) {
                unsigned long long xi, yi;
                rows(e, xi, yi);
#pragma unroll
                for (int j = 0; j < 3; j++) D[e][j] = ok(e) ? a.y[c][j][yi] - a.x[c][j][xi] : (T)0;
            }
            // multiply_a (replicated_3pc.h:44-67) of the bits with y - x, then
            // with x - y: z_p = r_p + s_p d_p + s_p d_q + s_q d_p
#pragma unroll 1  // one AES call in flight keeps the tile in registers
            for (int side = 0; side < 2; side++) {
                ORQ_NEXT_CALL();
#pragma unroll
                for (int e = 0; e < E; e++) {
                    if (!ok(e)) continue;
                    unsigned long long xi, yi;
                    rows(e, xi, yi);
#pragma unroll
                    for (int p = 0; p < 3; p++) {
                        const int q = (p + 1) % 3;
                        const T prod = bt[e][p] * D[e][p] + bt[e][p] * D[e][q] + bt[e][q] * D[e][p];
                        T* const v = side ? a.y[c][p] + yi : a.x[c][p] + xi;
                        *v += (K[e][(p + 2) % 3] - K[e][p]) + (side ? (T)0 - prod : prod);
                    }
                }
            }
        }
    }
}
#undef ORQ_NEXT_CALL

// BSharedVector::extend_lsb (b_shared_vector.h:145-147): every share becomes
// all ones where its LSB is set (local: repeating a bit is XOR-linear)
template <typename T>
__global__ void k_extend_lsb(CSh3 x, Sh3 y, unsigned long long n) {
    for (unsigned long long i = gtid(); i < n; i += gstride())
#pragma unroll
        for (int j = 0; j < 3; j++)
            reinterpret_cast<T*>(y.p[j])[i] = (T)0 - (reinterpret_cast<const T*>(x.p[j])[i] & 1);
}

// ---- bitonic sorting -----------------------------------------------------------
// One cooperative launch sorts one column or many: stage r of a bitonic network
// has the same box size and reversal for every size, so round r is a list of
// tiles (np pairs) of every item that still has a stage, and a grid barrier
// ends it. Item i's nonces at stage r are its base (where items 0..i-1 of the
// call end) plus r times its per-stage use, so the shares equal those of
// sequential calls. All threads compute a tile's keystream, for the round's
// first tile before the barrier is waited for; then each pair's thread runs
// the circuit. Bound by the T-table lookups, below 2^17 rows also by the
// barriers: 2^16 int32 rows took 136 launches, each staging 128 KB of tables,
// and 2.10 ms, and take 1.06 ms.
constexpr int kBitThreads = 512;
// pairs per tile: the keystream of 32 pairs is 3 KB (int32) or 6.75 KB. For
// int32 two tiles' worth is held, so that a tile costs one block barrier and
// the warps that are done with its circuit start on the next tile's keystream
// (2^20 rows: 23.6 and 21.1 ms); int64 keeps larger tiles instead (2^16 rows
// are then one tile an SM: 2.4 ms, and 3.4 with two buffers of 192 pairs).
template <int W>
constexpr int bitonic_max_pairs() { return W == 4 ? 512 : 448; }
template <int W>
constexpr int bitonic_bufs() { return W == 4 ? 2 : 1; }

struct BitonicItem {
    void* key[3];
    unsigned long long m;          // pairs (n / 2)
    unsigned long long nonce0[3];  // PAIR nonces at the item's first stage
    unsigned long long C, Cp;      // nonces per full / packed AND call
    uint32_t stages;
    int desc;
};

struct BitonicArgs {
    AesRK rk[3];
    BitonicItem one;           // the item of a call with one
    const BitonicItem* items;  // by stages, most first (null: `one`)
    const uint32_t* toff;      // [nitems + 1] tiles before each item
    uint32_t nitems, rounds, np;
    uint32_t* bar;             // arrivals, counted from 0
    int* err;
};

template <typename T>
__global__ void __launch_bounds__(kBitThreads, 1) k_bitonic(BitonicArgs a) {
    constexpr int W = sizeof(T);
    constexpr int L = cmp_levels<W>();
    constexpr uint32_t NFULL = L + 3;
    constexpr uint32_t WORDS = 32 * W / 4;  // keystream words per call and stream per warp
    constexpr uint32_t NB = 32 * W / 16;    // AES blocks of the same
    constexpr uint32_t PER = NFULL * 3 * NB;
    extern __shared__ __align__(16) uint32_t sm[];
    __shared__ __align__(16) uint32_t ksp2[2][kBitThreads / 128 + 1][3][4];  // packed call's block per 128 pairs
    __shared__ uint32_t ballots[kBitThreads / 32][3][3];
    __shared__ int s_dead;
    int flip = 0;
    aes_stage_tables(sm);
    const AesSmem S(sm);
    const uint32_t tid = threadIdx.x;
    const int lane = tid & 31, w = tid >> 5;
    const uint32_t G = gridDim.x, nw = a.np / 32;
    if (tid == 0) s_dead = 0;
    uint32_t target = 0, nact = a.nitems;
    int lev = 0, sub = 0;  // network round and substage
    for (uint32_t r = 0; r < a.rounds; r++) {
        const int hs = lev - sub;
        const bool first = sub == 0;
        if (a.items)
            while (nact > 1 && a.items[nact - 1].stages <= r) nact--;
        const uint32_t total = a.items ? a.toff[nact] : (uint32_t)ceil_div(a.one.m, a.np);
        bool waited = target == 0;
        // the previous round is complete everywhere
        const auto wait = [&]() {
            if (tid == 0) {
                // a cooperative launch's CTAs are all resident, so this ends; the
                // limit turns a lost arrival into an error
                uint32_t v, spins = 0;
                do {
                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.bar) : "memory");
                } while (v < target && ++spins < (1u << 24));
                if (v < target) {
                    atomicOr(a.err, kErrBarrier);
                    s_dead = 1;
                }
            }
        };
        for (uint32_t t = blockIdx.x; t < total; t += G, flip ^= bitonic_bufs<W>() - 1) {
            uint32_t* ksw = sm + kAesSmemBytes / 4 + flip * (nw * PER * 4);
            uint32_t(*ksp)[3][4] = ksp2[flip];
            uint32_t idx = 0, hi = nact - 1;  // item of tile t
            while (idx < hi) {
                const uint32_t mid = (idx + hi + 1) >> 1;
                if (a.toff[mid] <= t) idx = mid;
                else hi = mid - 1;
            }
            const BitonicItem& it = a.items ? a.items[idx] : a.one;
            const unsigned long long m = it.m, C = it.C, Cp = it.Cp;
            const unsigned long long base = (unsigned long long)(t - (a.items ? a.toff[idx] : 0u)) * a.np;
            const unsigned long long roff = (unsigned long long)r * ((L + 3) * C + Cp);
            const uint32_t wn = (uint32_t)min((unsigned long long)nw, ceil_div(m - base, 32));  // warps with pairs
            // this warp's pairs; past the round's first tile their rows are loaded
            // ahead of the keystream
            const bool mine = w < (int)nw;
            const unsigned long long p0w = base + 32 * w, p = p0w + lane;
            const bool valid = mine && p < m;
            unsigned long long xi, yi;
            bitonic_rows(p, hs, first, xi, yi);
            T* const* key = reinterpret_cast<T* const*>(it.key);
            T X[3] = {0, 0, 0}, Y[3] = {0, 0, 0};
            const auto rows = [&]() {
                if (valid)
#pragma unroll
                    for (int j = 0; j < 3; j++) {
                        X[j] = __ldcg(key[j] + xi);
                        Y[j] = __ldcg(key[j] + yi);
                    }
            };
            if (waited) rows();
            // a packed block covers 128 pairs: groups base / 128 on
            const uint32_t np3 = 3 * (((uint32_t)(base & 127) + 32 * wn + 127) / 128);
            for (uint32_t i = tid; i < np3 + wn * PER; i += kBitThreads) {
                uint32_t q;
                unsigned long long off, blk;
                uint32_t* o;
                if (i < np3) {
                    q = i % 3;
                    off = (unsigned long long)(L + 1) * C;
                    blk = base / 128 + i / 3;
                    o = ksp[i / 3][q];
                } else {
                    const uint32_t q2 = (i - np3) / PER, rem = (i - np3) - q2 * PER;
                    const uint32_t call = rem / (3 * NB);
                    q = (rem / NB) % 3;
                    off = call <= L ? call * C : call * C + Cp;  // the packed call is the (L + 2)nd
                    blk = (base + 32 * q2) * W / 16 + rem % NB;
                    o = ksw + q2 * PER * 4 + rem * 4;
                }
                *reinterpret_cast<uint4*>(o) = keystream_block_n(S, a.rk[q], it.nonce0[q] + roff + off, blk);
            }
            const bool late = !waited;
            if (late) wait();
            waited = true;
            __syncthreads();
            if (s_dead) return;  // uniform: written before the barrier above
            if (late) rows();
            if (mine) {  // (all warps of a packed word)
                T A[3], Bv[3], Sm[3], gt[3];
                // compare_rows: ASC compares x > y, DESC compares y > x
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    A[j] = it.desc ? Y[j] : X[j];
                    Bv[j] = it.desc ? X[j] : Y[j];
                }
                const uint32_t* myks = ksw + w * (NFULL * 3 * WORDS);
                const auto kword = [&](int call, int q) -> T {
                    const uint32_t* k = myks + (call * 3 + q) * WORDS;
                    if constexpr (W == 4) return (T)k[lane];
                    else return *reinterpret_cast<const T*>(k + 2 * lane);
                };
                bit_same3(A, Bv, kword, Sm);
                gt_bits3(A, Bv, Sm, valid, p, p0w, w, kword, ksp[p0w / 128 - base / 128], ballots, gt);
                // swap: x' = x ^ (ext(b) & (y ^ x)), y' = y ^ (ext(b) & (x ^ y))
                T E[3], D[3], K[3], Zx[3], Zy[3];
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    E[j] = gt[j] ? ~(T)0 : (T)0;
                    D[j] = X[j] ^ Y[j];
                    K[j] = kword(L + 1, j);
                }
                and3(E, D, K, Zx);
#pragma unroll
                for (int j = 0; j < 3; j++) K[j] = kword(L + 2, j);
                and3(E, D, K, Zy);
                if (valid)
#pragma unroll
                    for (int j = 0; j < 3; j++) {
                        key[j][xi] = X[j] ^ Zx[j];
                        key[j][yi] = Y[j] ^ Zy[j];
                    }
            }
            if constexpr (bitonic_bufs<W>() == 1) __syncthreads();  // the next tile rewrites the keystream
        }
        if (!waited) {  // a CTA without a tile still keeps step: arrivals are counted per round
            wait();
        }
        __syncthreads();
        if (s_dead) return;
        target += G;
        if (tid == 0) {
            __threadfence();
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
        }
        if (sub++ == lev) {
            lev++;
            sub = 0;
        }
    }
}

template <typename T, int MODE>
void launch_cmp(Ctx& c, const CmpArgs<T>& a, const char* name) {
    constexpr int W = sizeof(T), L = cmp_levels<W>();
    const auto kern = k_cmp<T, MODE>;
    constexpr int solo = kCmpSolo * cmp_calls<W, MODE>() * 3 * 32 * 16;
    ORQ_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kAesSmemBytes + solo));
    // a small call spreads over the SMs, a warp's pass each
    const unsigned long long units = ceil_div(a.m * W, 16);
    const unsigned grid = (unsigned)std::min<unsigned long long>(ceil_div(units, 32), (unsigned long long)c.num_sms);
    ProfScope ps(c, name, (MODE == 2 ? 9.0 : 12.0) * W * a.m,
                 3.0 * ((MODE == 2 ? L : L + 1) * (double)units + (MODE == 2 ? 0.0 : (double)ceil_div(a.m, 128))));
    const bool small = ceil_div(units, 32) <= (unsigned long long)grid * kCmpSolo;  // as the kernel's `solo`
    kern<<<grid, kAesThreads, kAesSmemBytes + (small ? solo : 0), c.stream>>>(a);
    ORQ_CUDA_CHECK(cudaGetLastError());
    c.kernels_launched++;
}

template <typename T>
void compare_t(Ctx& c, size_t n, CSh3 x, CSh3 y, Sh3 eq, Sh3 gt) {
    constexpr int W = sizeof(T);
    constexpr int L = cmp_levels<W>();
    CmpArgs<T> a{};
    for (int j = 0; j < 3; j++) {
        a.x[j] = (const T*)x.p[j];
        a.y[j] = (const T*)y.p[j];
        a.eq[j] = (T*)eq.p[j];
        a.gt[j] = (T*)gt.p[j];
        a.pair[j] = c.stream_arg(PAIR0 + j);
    }
    a.C = chunks_of((unsigned long long)n * W);
    a.Cp = chunks_of(ceil_div(n, 8 * W) * W);
    a.m = n;
    if (n) launch_cmp<T, 1>(c, a, "compare");
    for (int q = 0; q < 3; q++) c.nonce[PAIR0 + q] += (unsigned long long)(L + 1) * a.C + a.Cp;
}

// quicksort's compare of the rows at positions idx[0..n) with their segments' heads
// (quicksort.h:120-150): _compare's calls on the gathered rows, of which only
// the opened gt bits are written. The gathered copies, the eq and gt shares
// and the opened column that separate steps pass on are 400 bytes a row.
template <typename T>
void qs_compare_t(Ctx& c, size_t n, CSh3 rows, const uint32_t* ord, const uint32_t* idx, const int32_t* head, uint8_t* cb) {
    constexpr int W = sizeof(T);
    constexpr int L = cmp_levels<W>();
    CmpArgs<T> a{};
    for (int j = 0; j < 3; j++) {
        a.key[j] = (const T*)rows.p[j];
        a.pair[j] = c.stream_arg(PAIR0 + j);
    }
    a.ord = ord;
    a.idx = idx;
    a.head = head;
    a.cb = cb;
    a.C = chunks_of((unsigned long long)n * W);
    a.Cp = chunks_of(ceil_div(n, 8 * W) * W);
    a.m = n;
    if (n) launch_cmp<T, 3>(c, a, "compare");
    for (int q = 0; q < 3; q++) c.nonce[PAIR0 + q] += (unsigned long long)(L + 1) * a.C + a.Cp;
}

template <typename T>
void equal_t(Ctx& c, size_t n, CSh3 x, CSh3 y, Sh3 eq) {
    constexpr int W = sizeof(T);
    constexpr int L = cmp_levels<W>();
    CmpArgs<T> a{};
    for (int j = 0; j < 3; j++) {
        a.x[j] = (const T*)x.p[j];
        a.y[j] = (const T*)y.p[j];
        a.eq[j] = (T*)eq.p[j];
        a.pair[j] = c.stream_arg(PAIR0 + j);
    }
    a.C = chunks_of((unsigned long long)n * W);
    a.m = n;
    if (n) launch_cmp<T, 2>(c, a, "equal");
    for (int q = 0; q < 3; q++) c.nonce[PAIR0 + q] += (unsigned long long)L * a.C;
}

// not_b_1 (replicated_3pc.h:207): every share becomes !(s & 1)
template <typename T>
__global__ void k_not1(CSh3 x, Sh3 y, unsigned long long n) {
    for (unsigned long long i = gtid(); i < n; i += gstride())
#pragma unroll
        for (int j = 0; j < 3; j++)
            reinterpret_cast<T*>(y.p[j])[i] = (reinterpret_cast<const T*>(x.p[j])[i] & 1) ^ 1;
}

// Sorts `count` columns of power-of-two sizes in one launch; the shares of
// `count` calls in list order.
template <typename T>
void bitonic_t(Ctx& c, int count, const size_t* n, const Sh3* keys, const int* desc) {
    constexpr int W = sizeof(T);
    constexpr int L = cmp_levels<W>();
    std::vector<BitonicItem> items;
    unsigned long long off = 0, pairs = 0;
    double blocks = 0, bytes = 0;
    for (int i = 0; i < count; i++) {
        uint32_t k = 0;
        while (((size_t)1 << k) < n[i]) k++;
        if (!k) continue;
        BitonicItem it;
        it.m = n[i] / 2;
        it.C = chunks_of(it.m * W);
        it.Cp = chunks_of(ceil_div(it.m, 8ull * W) * W);
        it.stages = k * (k + 1) / 2;
        it.desc = desc[i];
        for (int j = 0; j < 3; j++) {
            it.key[j] = keys[i].p[j];
            it.nonce0[j] = c.nonce[PAIR0 + j] + off;
        }
        off += (unsigned long long)it.stages * ((L + 3) * it.C + it.Cp);
        pairs += it.m;
        blocks += it.stages * 3.0 * ((L + 3) * (double)ceil_div(it.m * W, 16) + (double)ceil_div(it.m, 128));
        bytes += it.stages * 12.0 * W * (double)it.m;
        items.push_back(it);
    }
    if (items.empty()) return;
    std::stable_sort(items.begin(), items.end(),
                     [](const BitonicItem& x, const BitonicItem& y) { return x.stages > y.stages; });
    // tiles that spread the first round over the SMs, whole packed words each
    constexpr unsigned long long step = 8 * W;
    const unsigned long long per_sm = ceil_div(pairs, (unsigned long long)c.num_sms);
    BitonicArgs a;
    a.np = (uint32_t)std::min<unsigned long long>(bitonic_max_pairs<W>(), ceil_div(per_sm, step) * step);
    for (int q = 0; q < 3; q++) a.rk[q] = c.rk[PAIR0 + q];
    a.one = items[0];
    a.nitems = (uint32_t)items.size();
    a.rounds = items[0].stages;
    a.items = nullptr;
    a.toff = nullptr;
    a.err = c.d_err;
    std::vector<uint32_t> toff(items.size() + 1, 0);
    for (size_t i = 0; i < items.size(); i++) toff[i + 1] = toff[i] + (uint32_t)ceil_div(items[i].m, a.np);
    const size_t ib = items.size() * sizeof(BitonicItem), tb = toff.size() * 4;
    std::unique_ptr<Scratch> table;
    if (items.size() > 1) {
        table.reset(new Scratch(c, ib + tb));
        uint8_t* h = (uint8_t*)c.batch_table(ib + tb);
        std::memcpy(h, items.data(), ib);
        std::memcpy(h + ib, toff.data(), tb);
        ORQ_CUDA_CHECK(cudaMemcpyAsync(table->p, h, ib + tb, cudaMemcpyHostToDevice, c.stream));
        ORQ_CUDA_CHECK(cudaEventRecord(c.batch.read, c.stream));
        a.items = table->as<BitonicItem>();
        a.toff = reinterpret_cast<const uint32_t*>(table->as<uint8_t>() + ib);
    }
    a.bar = c.grid_bar();
    ORQ_CUDA_CHECK(cudaMemsetAsync(a.bar, 0, 4, c.stream));
    constexpr size_t per_warp = (size_t)(L + 3) * 3 * (32 * W / 4) * 4;
    const size_t smem = kAesSmemBytes + bitonic_bufs<W>() * (a.np / 32) * per_warp;
    const auto kern = &k_bitonic<T>;
    ORQ_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)(kAesSmemBytes + bitonic_bufs<W>() * (bitonic_max_pairs<W>() / 32) * per_warp)));
    const unsigned grid = std::min<unsigned>(toff.back(), (unsigned)c.num_sms);
    {
        ProfScope ps(c, "bitonic", bytes, blocks);
        void* args[] = {&a};
        ORQ_CUDA_CHECK(cudaLaunchCooperativeKernel((const void*)kern, dim3(grid), dim3(kBitThreads), args, smem, c.stream));
    }
    c.kernels_launched++;
    for (int q = 0; q < 3; q++) c.nonce[PAIR0 + q] += off;
}

// nonces of one compare_rows over nkeys keys (each call of m pairs)
template <int W>
unsigned long long rows_cmp_nonces(int nkeys, unsigned long long C, unsigned long long Cp) {
    constexpr int L = cmp_levels<W>();
    return (unsigned long long)nkeys * ((L + 1) * C + Cp) + 2ull * (nkeys - 1) * C;
}

template <typename T>
void launch_rows_cmp(Ctx& c, const RowsCmpArgs<T>& a) {
    constexpr int W = sizeof(T);
    constexpr int L = cmp_levels<W>();
    constexpr int kThreads = cmp_threads<W>();
    const unsigned long long per_sm = ceil_div(a.m, (unsigned long long)c.num_sms);
    const int nt = (int)std::min<unsigned long long>(kThreads, std::max<unsigned long long>(64, ceil_div(per_sm, 64) * 64));
    const size_t per_warp = (size_t)(L + 3) * 3 * (32 * W / 4) * 4;
    const size_t smem = kAesSmemBytes + (size_t)(nt / 32) * per_warp;
    auto kern = k_rows_cmp<T>;
    ORQ_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)(kAesSmemBytes + (size_t)(kThreads / 32) * per_warp)));
    const unsigned long long units = ceil_div(a.m, (unsigned long long)nt);
    const unsigned grid = (unsigned)std::min<unsigned long long>(units ? units : 1, (unsigned long long)c.num_sms);
    const double full_calls = (double)a.nkeys * (L + 1) + 2.0 * (a.nkeys - 1);
    ProfScope ps(c, "compare_rows", (6.0 * a.nkeys + 3.0) * W * a.m,
                 full_calls * 3.0 * ceil_div(a.m * W, 16) + 3.0 * a.nkeys * ceil_div(ceil_div(a.m, 8 * W) * W, 16));
    kern<<<grid, nt, smem, c.stream>>>(a);
    ORQ_CUDA_CHECK(cudaGetLastError());
    c.kernels_launched++;
}

// launches one swap and returns the nonces it used: two calls per column and
// three for the b2a of the bits
template <typename T>
unsigned long long launch_rows_swap(Ctx& c, const RowsSwapArgs<T>& a) {
    constexpr int W = sizeof(T);
    const unsigned long long calls = 2ull * (a.nbool + a.narith) + (a.b2a && a.narith ? 3ull : 0ull);
    if (a.m && (a.nbool + a.narith))
        launch_aes(c, "swap", (12.0 * (a.nbool + a.narith) + 3.0) * W * a.m,
                   3.0 * calls * ceil_div(a.m * W, 16), k_rows_swap<T>, ceil_div(a.m, (unsigned long long)(16 / W)), a);
    return calls * a.C;
}

template <typename T>
void compare_rows_t(Ctx& c, size_t n, int nkeys, const CSh3* x, const CSh3* y, const int* desc, Sh3 gt) {
    constexpr int W = sizeof(T);
    RowsCmpArgs<T> a{};
    for (int k = 0; k < nkeys; k++) {
        for (int j = 0; j < 3; j++) {
            a.x[k][j] = (const T*)x[k].p[j];
            a.y[k][j] = (const T*)y[k].p[j];
        }
        a.desc[k] = desc[k] != 0;
    }
    for (int j = 0; j < 3; j++) {
        a.gt[j] = (T*)gt.p[j];
        a.pair[j] = c.stream_arg(PAIR0 + j);
    }
    a.nkeys = nkeys;
    a.m = n;
    a.hs = -1;
    a.C = chunks_of((unsigned long long)n * W);
    a.Cp = chunks_of(ceil_div(n, 8 * W) * W);
    if (n) launch_rows_cmp(c, a);
    for (int q = 0; q < 3; q++) c.nonce[PAIR0 + q] += rows_cmp_nonces<W>(nkeys, a.C, a.Cp);
}

template <typename T>
void swap_t(Ctx& c, size_t n, bool arith, int ncols, const Sh3* x, const Sh3* y, CSh3 bits) {
    constexpr int W = sizeof(T);
    RowsSwapArgs<T> a{};
    for (int k = 0; k < ncols; k++)
        for (int j = 0; j < 3; j++) {
            a.x[k][j] = (T*)x[k].p[j];
            a.y[k][j] = (T*)y[k].p[j];
        }
    for (int j = 0; j < 3; j++) {
        a.bits[j] = (const T*)bits.p[j];
        a.pair[j] = c.stream_arg(PAIR0 + j);
    }
    a.nbool = arith ? 0 : ncols;
    a.narith = arith ? ncols : 0;
    a.m = n;
    a.hs = -1;
    a.C = chunks_of((unsigned long long)n * W);
    const unsigned long long used = launch_rows_swap(c, a);
    for (int q = 0; q < 3; q++) c.nonce[PAIR0 + q] += used;
}

// bitonic_sort (operators/sorting.h:266-353) over several key columns with
// A- and B-shared data columns: per stage one compare_rows launch writes the
// comparison bits, one swap launch moves keys, B data and (through b2a_bit of
// the bits) A data.
template <typename T>
void bitonic_rows_t(Ctx& c, size_t n, int nkeys, const Sh3* keys, const int* desc, int na,
                    const Sh3* data_a, int nb, const Sh3* data_b) {
    constexpr int W = sizeof(T);
    int rounds = 0;
    while (((size_t)1 << rounds) < n) rounds++;
    const size_t m = n / 2;
    Scratch bits(c, 3 * m * W);
    RowsCmpArgs<T> ca{};
    RowsSwapArgs<T> sa{};
    for (int k = 0; k < nkeys; k++) {
        for (int j = 0; j < 3; j++) {
            ca.x[k][j] = ca.y[k][j] = (const T*)keys[k].p[j];
            sa.x[k][j] = sa.y[k][j] = (T*)keys[k].p[j];
        }
        ca.desc[k] = desc[k] != 0;
    }
    for (int k = 0; k < nb; k++)
        for (int j = 0; j < 3; j++) sa.x[nkeys + k][j] = sa.y[nkeys + k][j] = (T*)data_b[k].p[j];
    for (int k = 0; k < na; k++)
        for (int j = 0; j < 3; j++) sa.x[nkeys + nb + k][j] = sa.y[nkeys + nb + k][j] = (T*)data_a[k].p[j];
    for (int j = 0; j < 3; j++) {
        ca.gt[j] = bits.as<T>() + j * m;
        sa.bits[j] = bits.as<T>() + j * m;
    }
    ca.nkeys = nkeys;
    ca.m = sa.m = m;
    ca.C = sa.C = chunks_of((unsigned long long)m * W);
    ca.Cp = chunks_of(ceil_div(m, 8 * W) * W);
    sa.nbool = nkeys + nb;
    sa.narith = na;
    sa.b2a = 1;
    for (int i = 0; i < rounds; i++)
        for (int jj = 0; jj <= i; jj++) {
            ca.hs = sa.hs = i - jj;
            ca.first = sa.first = jj == 0;
            for (int q = 0; q < 3; q++) ca.pair[q] = c.stream_arg(PAIR0 + q);
            launch_rows_cmp(c, ca);
            for (int q = 0; q < 3; q++) c.nonce[PAIR0 + q] += rows_cmp_nonces<W>(nkeys, ca.C, ca.Cp);
            for (int q = 0; q < 3; q++) sa.pair[q] = c.stream_arg(PAIR0 + q);
            const unsigned long long used = launch_rows_swap(c, sa);
            for (int q = 0; q < 3; q++) c.nonce[PAIR0 + q] += used;
        }
}

template <typename T>
void extend_lsb_t(Ctx& c, size_t n, CSh3 x, Sh3 y) {
    if (!n) return;
    ProfScope ps(c, "extend_lsb", 6.0 * sizeof(T) * n);
    k_extend_lsb<T><<<plain_grid(c, n), 256, 0, c.stream>>>(x, y, n);
    ORQ_CUDA_CHECK(cudaGetLastError());
    c.kernels_launched++;
}

}  // namespace

void op_compare_rows(Ctx& c, int w, size_t n, int nkeys, const CSh3* x, const CSh3* y, const int* desc, Sh3 gt) {
    if (nkeys < 1 || nkeys > kMaxRowKeys) throw std::invalid_argument("compare_rows takes 1 to 8 key columns");
    if (w == 4) compare_rows_t<uint32_t>(c, n, nkeys, x, y, desc, gt);
    else if (w == 8) compare_rows_t<unsigned long long>(c, n, nkeys, x, y, desc, gt);
    else throw std::invalid_argument("compare_rows supports int32 and int64 keys");
}

void op_swap(Ctx& c, int w, size_t n, bool arith, int ncols, const Sh3* x, const Sh3* y, CSh3 bits) {
    if (ncols < 0 || ncols > kMaxRowCols) throw std::invalid_argument("swap takes 0 to 40 column pairs");
    if (w == 4) swap_t<uint32_t>(c, n, arith, ncols, x, y, bits);
    else if (w == 8) swap_t<unsigned long long>(c, n, arith, ncols, x, y, bits);
    else throw std::invalid_argument("swap supports 4 and 8-byte shares");
}

void op_extend_lsb(Ctx& c, int w, size_t n, CSh3 x, Sh3 y) {
    if (w == 4) extend_lsb_t<uint32_t>(c, n, x, y);
    else if (w == 8) extend_lsb_t<unsigned long long>(c, n, x, y);
    else throw std::invalid_argument("extend_lsb supports 4 and 8-byte shares");
}

void op_bitonic_sort_rows(Ctx& c, int w, size_t n, int nkeys, const Sh3* keys, const int* desc, int na,
                          const Sh3* data_a, int nb, const Sh3* data_b) {
    if (n & (n - 1)) throw std::invalid_argument("bitonic sort needs a power-of-two size");
    if (nkeys < 1 || nkeys > kMaxRowKeys) throw std::invalid_argument("bitonic sort takes 1 to 8 key columns");
    if (na < 0 || nb < 0 || nkeys + na + nb > kMaxRowCols)
        throw std::invalid_argument("bitonic sort takes at most 40 key and data columns");
    if (w != 4 && w != 8) throw std::invalid_argument("bitonic sort supports int32 and int64 keys");
    if (n < 2) return;
    if (nkeys == 1 && na == 0 && nb == 0) {  // one launch for the whole sort
        op_bitonic_sort(c, w, n, keys[0], desc[0] != 0);
        return;
    }
    if (w == 4) bitonic_rows_t<uint32_t>(c, n, nkeys, keys, desc, na, data_a, nb, data_b);
    else bitonic_rows_t<unsigned long long>(c, n, nkeys, keys, desc, na, data_a, nb, data_b);
}

void op_compare(Ctx& c, int w, size_t n, CSh3 x, CSh3 y, Sh3 eq, Sh3 gt) {
    if (w == 4) compare_t<uint32_t>(c, n, x, y, eq, gt);
    else if (w == 8) compare_t<unsigned long long>(c, n, x, y, eq, gt);
    else if (w == 16) compare_t<unsigned __int128>(c, n, x, y, eq, gt);
    else throw std::invalid_argument("compare supports 4, 8 and 16-byte keys");
}

void op_qs_compare(Ctx& c, int w, size_t n, CSh3 rows, const uint32_t* ord, const uint32_t* idx, const int32_t* head,
                   uint8_t* cb) {
    if (w == 16) qs_compare_t<unsigned __int128>(c, n, rows, ord, idx, head, cb);
    else if (w == 8) qs_compare_t<unsigned long long>(c, n, rows, ord, idx, head, cb);
    else throw std::invalid_argument("quicksort rows are 8 or 16 bytes");
}
void op_equal(Ctx& c, int w, size_t n, CSh3 x, CSh3 y, Sh3 eq) {
    if (w == 4) equal_t<uint32_t>(c, n, x, y, eq);
    else if (w == 8) equal_t<unsigned long long>(c, n, x, y, eq);
    else if (w == 16) equal_t<unsigned __int128>(c, n, x, y, eq);
    else throw std::invalid_argument("equality supports 4, 8 and 16-byte keys");
}

void op_not1(Ctx& c, int w, size_t n, CSh3 x, Sh3 y) {
    if (!n) return;
    const unsigned g = plain_grid(c, n);
    ProfScope ps(c, "not_b_1", 6.0 * w * n);
    if (w == 4) k_not1<uint32_t><<<g, 256, 0, c.stream>>>(x, y, n);
    else if (w == 8) k_not1<unsigned long long><<<g, 256, 0, c.stream>>>(x, y, n);
    else throw std::invalid_argument("not_b_1 supports 4 and 8-byte shares");
    ORQ_CUDA_CHECK(cudaGetLastError());
    c.kernels_launched++;
}

void op_bitonic_sort(Ctx& c, int w, size_t n, Sh3 key, bool desc) {
    if (n & (n - 1)) throw std::invalid_argument("bitonic sort needs a power-of-two size");
    if (n < 2) return;
    const int d = desc;
    op_bitonic_sort_batch(c, w, 1, &n, &key, &d);
}
void op_bitonic_sort_batch(Ctx& c, int w, int count, const size_t* n, const Sh3* keys, const int* desc) {
    if (w == 4) bitonic_t<uint32_t>(c, count, n, keys, desc);
    else if (w == 8) bitonic_t<unsigned long long>(c, count, n, keys, desc);
    else throw std::invalid_argument("bitonic sort supports int32 and int64 keys");
}

}  // namespace orqcu
