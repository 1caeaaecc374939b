// fy.cu — generation of sharded permutations: Fisher–Yates from the group
// PRGs, bit-exact with ORQ.
//
// Generation restates gen_perm (include/core/random/permutations/
// hm_sharded_permutation_generator.h:70-108): draws are u32 words of the group
// stream taken from getNext buffers of 2^20 words (4 nonces each), reduced by
// mask = 2^bit_width(n) - 1; draw values above n-1-i are rejected; the i-th
// accepted value v gives swap(p[i], p[i+v]). A permutation starts on a fresh
// buffer, so consecutive permutations of one group form a chain whose start
// nonces depend on how many draws the previous one used.
//
// GPU design:
//  * the draws of a group's buffers do not depend on where permutations start,
//    so k_fy_gen computes them ahead, as pure keystream, into a ring;
//  * a permutation's threshold T = n-1-i falls along a predictable curve
//    (x' = -x/M), so k_fy_classify decides almost every draw in parallel from a
//    window around the curve: accepted, rejected, or uncertain;
//  * k_fy_resolve (one CTA per group) walks only the uncertain draws in order,
//    and k_fy_emit writes the accepted offsets at their exact ranks and checks
//    the windows against the exact thresholds;
//    a one-CTA scanner that replayed every draw bounded the chain before (the
//    same radix steps with it and without: 2^22 rows 418 and 280 ms, 2^20 rows
//    127.6 and 62.8, 100003 rows 19.0 and 12.5; the faster bit loop and the rest
//    have since made 214, 53 and 6.6 of these);
//  * fy_small (M <= 2^15, many of M = 2^16; one buffer per permutation almost always):
//    every (permutation, group) in its own CTA at once from predicted start
//    buffers, re-run from the first wrong prediction until all are verified;
//  * fy_finalize: turns the accepted offsets into the inverse permutation in
//    parallel (the gather index of an application; the permutation itself,
//    which only inverse applications read, is derived when one asks for it).
#include <algorithm>
#include <cstring>
#include <memory>

#include "launch.cuh"

namespace orqcu {

namespace {

// ---------------------------------------------------------------------------
// The chain of permutations of one group (M = 2^bit_width(n) >= 2^16).
constexpr uint32_t kBufDraws = 1u << 20;   // draws per getNext buffer
constexpr uint32_t kListDraws = 2048;      // draws behind one sparse list
constexpr uint32_t kListCap = 256;
constexpr uint32_t kListsPerBuf = kBufDraws / kListDraws;
constexpr uint32_t kRuns = 8;              // runs (warps) per tile; a CTA classifies a tile
constexpr uint32_t kMaxRunLists = 4;       // a run is 1..4 lists' draws (FyScanArgs::rl)
constexpr uint32_t kRunUnc = 512;          // uncertain draws kept per run
constexpr uint32_t kTileUnc = kRuns * kRunUnc;
constexpr uint32_t kPieceUnc = 8192;       // uncertain draws k_fy_resolve holds at once
constexpr int kGenThreads = 512;
constexpr int kTabEntries = 520;           // U[256], V[257] of one chunk, padded

constexpr uint32_t kMissed = 1;    // a window missed its threshold
constexpr uint32_t kOverflow = 2;  // more uncertain draws in a run than it keeps

// Scan state of one group's chain. `pos` counts tiles and `start` buffers from
// the chain's first buffer.
struct FyState {
    unsigned long long pos;    // first tile not yet scanned
    unsigned long long start;  // buffer where the current permutation starts
    uint32_t m;                // index of the current permutation
    uint32_t i;                // accepted so far
    uint32_t done;             // every permutation is complete
    uint32_t bad;              // kMissed, kOverflow
};

// GCM's counter block is (nonce, 0, BE32(j + 2)): inside a chunk of 65536
// blocks only the counter's low bytes change, and after two AES rounds the
// state is U[ctr & 255] ^ V[ctr >> 8] with tables that depend on the key and
// the chunk's nonce alone (byte 15 reaches column 0 of round 1, the other
// counter bytes columns 1 and 2; round 2 is the XOR of one table word per
// column). Two loads replace 32 of a block's 224 lookups: alone in a loop, the
// keystream goes from 4.17e10 to 4.70e10 blocks/s.
__global__ void __launch_bounds__(544) k_fy_tab(StreamArg st, uint4* tab) {
    const auto T = [](int t, uint32_t w, int byte) { return __ldg(&g_aes_T[t * 256 + ((w >> (8 * byte)) & 255u)]); };
    const AesRK& rk = st.rk;
    const unsigned long long nonce = st.nonce + blockIdx.x;
    uint4* out = tab + (size_t)blockIdx.x * kTabEntries;
    const uint32_t w0 = (uint32_t)nonce ^ rk.k[0], w1 = (uint32_t)(nonce >> 32) ^ rk.k[1], w2 = rk.k[2];
    const uint32_t t = threadIdx.x;
    if (t < 256) {
        const uint32_t w3 = (t << 24) ^ rk.k[3];
        const uint32_t n0 = T(0, w0, 0) ^ T(1, w1, 1) ^ T(2, w2, 2) ^ T(3, w3, 3) ^ rk.k[4];
        out[t] = make_uint4(T(0, n0, 0), T(3, n0, 3), T(2, n0, 2), T(1, n0, 1));
    } else if (t < 513) {
        const uint32_t w3 = __byte_perm((t - 256) << 8, 0, 0x0123) ^ rk.k[3];
        const uint32_t n1 = T(0, w1, 0) ^ T(1, w2, 1) ^ T(2, w3, 2) ^ T(3, w0, 3) ^ rk.k[5];
        const uint32_t n2 = T(0, w2, 0) ^ T(1, w3, 1) ^ T(2, w0, 2) ^ T(3, w1, 3) ^ rk.k[6];
        const uint32_t n3 = T(0, w3, 0) ^ T(1, w0, 1) ^ T(2, w1, 2) ^ T(3, w2, 3) ^ rk.k[7];
        out[t] = make_uint4(T(1, n1, 1) ^ T(2, n2, 2) ^ T(3, n3, 3) ^ rk.k[8],
                            T(0, n1, 0) ^ T(1, n2, 1) ^ T(2, n3, 2) ^ rk.k[9],
                            T(0, n2, 0) ^ T(1, n3, 1) ^ T(3, n1, 3) ^ rk.k[10],
                            T(0, n3, 0) ^ T(2, n1, 2) ^ T(3, n2, 3) ^ rk.k[11]);
    }
}

struct FyGenArgs {
    StreamArg st;
    const uint4* tab;  // k_fy_tab of the same buffers
    uint32_t mask, th; // th: draws below it go to the sparse lists
    uint32_t lists;    // sparse lists (kListDraws draws each) to produce
    uint32_t* raw;     // masked draws
    uint32_t* lst;     // [lists][kListCap]
    uint32_t* lcnt;    // [lists] entries; above kListCap: the list overflowed
    const FyState* state;
};

// Masked draws of a range of buffers, and per kListDraws of them the list of
// those below n/16 in draw order (what the scan of a permutation's last 7/8 of
// draws reads). A warp owns a list, so nothing but the table staging is
// block-wide. Bound by the T-table lookups (shared-memory pipe): 192 lookups,
// two table loads and one 16-byte store a block; 64 buffers take 414 us
// (4.06e10 blocks/s; with nested lists built by block scans it was 2.0e10).
__global__ void __launch_bounds__(kGenThreads, 1) k_fy_gen(FyGenArgs a) {
    extern __shared__ __align__(16) uint32_t sm[];
    aes_stage_tables(sm);
    const AesSmem S(sm);
    if (*(volatile const uint32_t*)&a.state->done) return;  // no barrier follows
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t nw = gridDim.x * (kGenThreads / 32);
    constexpr uint32_t kPerChunk = 65536 / (kListDraws / 4);  // lists per chunk
    for (uint32_t l = blockIdx.x * (kGenThreads / 32) + (threadIdx.x >> 5); l < a.lists; l += nw) {
        const uint4* U = a.tab + (size_t)(l / kPerChunk) * kTabEntries;
        const uint4* V = U + 256;
        uint32_t ctr = (l % kPerChunk) * (kListDraws / 4) + lane + 2;
        uint4* out = reinterpret_cast<uint4*>(a.raw + (size_t)l * kListDraws) + lane;
        uint32_t* li = a.lst + (size_t)l * kListCap;
        uint32_t lc = 0;
        uint4 u = __ldg(U + (ctr & 255u)), v = __ldg(V + (ctr >> 8));
#pragma unroll 1
        for (int it = 0; it < (int)(kListDraws / 128); it++) {
            uint32_t s0 = u.x ^ v.x, s1 = u.y ^ v.y, s2 = u.z ^ v.z, s3 = u.w ^ v.w;
            ctr += 32;
            if (it + 1 < (int)(kListDraws / 128)) {
                u = __ldg(U + (ctr & 255u));
                v = __ldg(V + (ctr >> 8));
            }
            aes256_rounds_from<3>(S, a.st.rk, s0, s1, s2, s3);
            s0 &= a.mask;
            s1 &= a.mask;
            s2 &= a.mask;
            s3 &= a.mask;
            out[32 * it] = make_uint4(s0, s1, s2, s3);
            const bool c0 = s0 < a.th, c1 = s1 < a.th, c2 = s2 < a.th, c3 = s3 < a.th;
            const uint32_t b0 = __ballot_sync(0xffffffffu, c0), b1 = __ballot_sync(0xffffffffu, c1);
            const uint32_t b2 = __ballot_sync(0xffffffffu, c2), b3 = __ballot_sync(0xffffffffu, c3);
            uint32_t o = lc + __popc(b0 & lt) + __popc(b1 & lt) + __popc(b2 & lt) + __popc(b3 & lt);
            lc += __popc(b0) + __popc(b1) + __popc(b2) + __popc(b3);
            if (lc <= kListCap) {
                if (c0) li[o++] = s0;
                if (c1) li[o++] = s1;
                if (c2) li[o++] = s2;
                if (c3) li[o] = s3;
            }
        }
        if (lane == 0) a.lcnt[l] = lc;
    }
}

// One run's classification (k_fy_classify -> k_fy_emit).
struct FyRun {
    uint32_t cpre, upre;  // certain / uncertain draws of the tile before the run
    uint32_t cnt, unc;    // candidates (certain + uncertain) and uncertain draws
    long long lo, hi;     // the window that T at the run's start was assumed in
};
struct FySeg {  // what k_fy_resolve settled of a step, for k_fy_emit
    uint32_t ntiles, m;
};

struct FyScanArgs {
    uint32_t n, count, g;
    uint32_t mbits;                // M = 2^mbits
    uint32_t th;                   // list threshold of k_fy_gen
    uint32_t rl;                   // lists per run: 1, 2 or 4
    uint32_t tpb;                  // tiles per buffer: kListsPerBuf / (kRuns * rl)
    uint32_t ring_tiles;           // tiles the ring holds
    uint32_t seg_cap;              // tiles a step may scan
    unsigned long long limit;      // tiles generated so far
    double rate;                   // log(1 - 1/M)
    double width;                  // window half-width in standard deviations
    const uint32_t *raw, *lst, *lcnt;
    FyState* state;
    uint32_t* cand;                // [seg_cap][kRuns][rl * kListDraws] candidates
    uint2* unc;                    // [seg_cap][kTileUnc] (v + certain draws before it in the tile, place in its run's candidates)
    FyRun* run;                    // [seg_cap][kRuns]
    uint32_t *tc, *tu;             // [seg_cap] certain / uncertain draws
    uint32_t* base;                // [seg_cap] rank of the tile's first acceptance
    uint32_t* uoff;                // [seg_cap] index of the tile's first uncertain draw in `ok`
    uint32_t* ok;                  // one bit per uncertain draw of the step: accepted
    FySeg* seg;
    uint32_t* acc;                 // [count][3][n] accepted offsets
};

// Tiles of the next step: what is generated, at most seg_cap, and not much
// past the place where the permutation ends (x = n - i values remain; they
// take about M (ln x + 4) draws or fewer with probability 0.98; a step that
// stops short is continued by the next). Integer arithmetic, so that every
// kernel of the step finds the same number. `bad` is no part of it: another
// CTA's classification may set it while this one's warps read the state, and
// warps with different numbers would take sums of shared memory that the others
// have not written, and store by them.
__device__ __forceinline__ uint32_t fy_step_tiles(const FyScanArgs& a, const FyState& s) {
    if (s.done || s.pos >= a.limit) return 0;
    const uint32_t lg = 32 - __clz(a.n - s.i);                                // log2(x) rounded up
    // M in tiles (kRuns * rl * 2048 draws each), times ln x + 4 in 16 fractional bits
    const unsigned long long span =
        ((((1ull << a.mbits) / (kRuns * a.rl * kListDraws)) * (lg * 45427ull + 4 * 65536ull)) >> 16) + 2;
    unsigned long long t = a.limit - s.pos;
    t = t < a.seg_cap ? t : a.seg_cap;
    return (uint32_t)(t < span ? t : span);
}

// Classification of one step's draws. `x` values remain when the step begins,
// so after d draws x e^(d log(1-1/M)) remain on average, with variance below
// x p (1 - p): T at a run's start lies in [lo, hi] = mean -+ (width sigma + 3
// width) except about once in 1e7 permutations (checked afterwards). With k
// candidates and c certain draws of the run before draw q: accepted for
// certain if v + k <= lo (at most k acceptances so far), rejected if v > hi - c
// (at least c), uncertain otherwise. Sizes: 2^22 rows have ~1e3 deviations at
// worst, so ~1.5 in 1000 draws are uncertain. Small register count: the CTAs
// run beside the generator's, in its idle issue slots.
__global__ void __launch_bounds__(kRuns * 32, 4) k_fy_classify(FyScanArgs a) {
    __shared__ uint2 su[kRuns][kRunUnc];
    __shared__ uint32_t scert[kRuns], sunc[kRuns];
    const FyState s = *a.state;
    const uint32_t nt = fy_step_tiles(a, s);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const double x = (double)(a.n - s.i);
    const uint32_t rd = a.rl * kListDraws;  // draws per run
    for (uint32_t t = blockIdx.x; t < nt; t += gridDim.x) {
        const uint32_t rt = (uint32_t)((s.pos + t) % a.ring_tiles);
        const double p = exp(a.rate * ((double)t * kRuns + (double)w) * rd);
        const double half = a.width * sqrt(x * p * (1.0 - p)) + 3.0 * a.width;
        const long long lo = (long long)floor(x * p - 1.0 - half);
        const long long hi = min((long long)ceil(x * p - 1.0 + half), (long long)(a.n - s.i) - 1);
        const bool some = lo >= 0;
        const uint32_t lou = some ? (uint32_t)lo : 0u, hiu = (uint32_t)hi;
        const size_t l0 = ((size_t)rt * kRuns + w) * a.rl;
        const uint32_t* raw = a.raw + l0 * kListDraws;
        uint32_t* cand = a.cand + ((size_t)t * kRuns + w) * rd;
        uint32_t k = 0, nu = 0;
        const uint32_t mycnt = lane < (int)a.rl ? a.lcnt[l0 + lane] : 0u;
        // (q, e): list q of the run, first of the next 128 entries in it
        const auto source = [&](uint32_t q, const uint32_t*& src, uint32_t& cnt) {
            const uint32_t c = __shfl_sync(0xffffffffu, mycnt, q & (kMaxRunLists - 1));
            const bool use = hiu < a.th && c <= kListCap;
            src = use ? a.lst + (l0 + q) * kListCap : raw + q * kListDraws;
            cnt = use ? c : kListDraws;
        };
        const uint32_t* src;
        uint32_t cnt;
        source(0, src, cnt);
        uint32_t q = 0, e = 0;
        // three chunks of 128 entries in flight; left: entries of a chunk
        constexpr int kAhead = 3;
        uint4 nx[kAhead];
        uint32_t left[kAhead];
        const auto next = [&](uint4& x, uint32_t& l) {
            l = 0;
            if (q >= a.rl) return;
            if (e + 4 * lane < cnt) x = *reinterpret_cast<const uint4*>(src + e + 4 * lane);
            l = cnt - e < 128 ? cnt - e : 128;
            e += 128;
            while (e >= cnt) {  // (an empty list holds no chunk)
                if (++q >= a.rl) break;
                e = 0;
                source(q, src, cnt);
                if (cnt) break;
            }
        };
        while (cnt == 0 && ++q < a.rl) source(q, src, cnt);
#pragma unroll
        for (int i = 0; i < kAhead; i++) {
            nx[i] = make_uint4(0, 0, 0, 0);
            next(nx[i], left[i]);
        }
        while (left[0]) {
            const uint4 v4 = nx[0];
            const uint32_t n4 = left[0];
#pragma unroll
            for (int i = 0; i + 1 < kAhead; i++) {
                nx[i] = nx[i + 1];
                left[i] = left[i + 1];
            }
            next(nx[kAhead - 1], left[kAhead - 1]);
            const uint32_t v[4] = {v4.x, v4.y, v4.z, v4.w};
            const uint32_t c = k - nu;
            bool cd[4], un[4];
            uint32_t m[4];
            bool any = false;
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const uint32_t j = 4u * lane + r;
                cd[r] = j < n4 && v[r] + c <= hiu;
                un[r] = cd[r] && !(some && v[r] + k + j <= lou);
                any = any || un[r];
                m[r] = __ballot_sync(0xffffffffu, cd[r]);
            }
            uint32_t o = k + __popc(m[0] & lt) + __popc(m[1] & lt) + __popc(m[2] & lt) + __popc(m[3] & lt);
            uint32_t po[4];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                po[r] = o;
                if (cd[r]) cand[o++] = v[r];
            }
            if (__any_sync(0xffffffffu, any)) {
                uint32_t um[4];
#pragma unroll
                for (int r = 0; r < 4; r++) um[r] = __ballot_sync(0xffffffffu, un[r]);
                uint32_t uo = nu + __popc(um[0] & lt) + __popc(um[1] & lt) + __popc(um[2] & lt) + __popc(um[3] & lt);
#pragma unroll
                for (int r = 0; r < 4; r++)
                    if (un[r]) {
                        if (uo < kRunUnc) su[w][uo] = make_uint2(v[r] + (po[r] - uo), po[r]);
                        uo++;
                    }
                nu += __popc(um[0]) + __popc(um[1]) + __popc(um[2]) + __popc(um[3]);
            }
            k += __popc(m[0]) + __popc(m[1]) + __popc(m[2]) + __popc(m[3]);
        }
        if (nu > kRunUnc) {
            if (lane == 0) atomicOr(&a.state->bad, kOverflow);
            nu = kRunUnc;
        }
        if (lane == 0) {
            scert[w] = k - nu;
            sunc[w] = nu;
        }
        __syncthreads();
        uint32_t cp = 0, up = 0, ct = 0, ut = 0;
        for (uint32_t r = 0; r < kRuns; r++) {
            if ((int)r < w) {
                cp += scert[r];
                up += sunc[r];
            }
            ct += scert[r];
            ut += sunc[r];
        }
        uint2* ou = a.unc + (size_t)t * kTileUnc + up;
        for (uint32_t j = lane; j < nu; j += 32) {
            const uint2 z = su[w][j];
            ou[j] = make_uint2(z.x + cp, z.y);
        }
        if (lane == 0) a.run[(size_t)t * kRuns + w] = FyRun{cp, up, k, nu, lo, hi};
        if (threadIdx.x == 0) {
            a.tc[t] = ct;
            a.tu[t] = ut;
        }
        __syncthreads();
    }
}

// Decides a step's uncertain draws (one CTA), gives every tile the rank of its
// first acceptance, and moves the state to the next step. An uncertain draw
// with v + (certain draws before it) = u is accepted iff u <= X - a, a the
// uncertain acceptances before it. A thread holds kResEach consecutive ones and
// decides them from an assumed a at its first; the block's prefix sums give the
// next assumption, until nothing changes: thread 0 starts from the true count,
// so the fixed point is the sequential result, and each pass shrinks the error
// about tenfold (a piece's threshold moves by much less than the window).
// Between launches of a group's stream nothing else writes the state but the
// flag `bad`.
constexpr int kResThreads = 512;
constexpr int kResEach = kPieceUnc / kResThreads;  // 16
__global__ void __launch_bounds__(kResThreads, 1) k_fy_resolve(FyScanArgs a) {
    // entry k at k + k / 16: a thread reads its 16 without bank conflicts
    __shared__ uint32_t su[kPieceUnc + kPieceUnc / kResEach];
    __shared__ uint32_t smask[kResThreads], sbef[kResThreads + 1];
    __shared__ uint32_t sc[kResThreads], so[kResThreads + 1];
    __shared__ uint32_t red[33];
    __shared__ uint32_t s_take, s_end, s_call;
    const FyState s = *a.state;
    const uint32_t nt = s.bad ? 0 : fy_step_tiles(a, s);  // (nothing else runs that sets it)
    const uint32_t tid = threadIdx.x;
    if (!nt) {
        if (tid == 0) *a.seg = FySeg{0, s.m};
        return;
    }
    const int top = (int)(a.n - s.i - 1);  // T when the step begins
    uint32_t cbase = 0, abase = 0;         // certain / uncertain acceptances of earlier pieces
    uint32_t t_end = 0xffffffffu, words = 0;
    for (uint32_t t0 = 0; t0 < nt && t_end == 0xffffffffu;) {
        // the next tiles whose uncertain draws fit the piece
        const uint32_t t = t0 + tid;
        const uint32_t c = t < nt ? a.tc[t] : 0u, u = t < nt ? min(a.tu[t], kTileUnc) : 0u;
        uint32_t ctot, utot;
        const uint32_t cpre = block_excl_sum(c, red, ctot);
        const uint32_t upre = block_excl_sum(u, red, utot);
        sc[tid] = cpre;
        so[tid] = upre;
        if (tid == 0) {
            s_take = 0;
            s_end = 0xffffffffu;
        }
        __syncthreads();
        if (t < nt && upre + u <= kPieceUnc) atomicMax(&s_take, tid + 1);
        __syncthreads();
        const uint32_t take = s_take;
        if (tid == take - 1) {
            so[take] = upre + u;
            s_call = cpre + c;
        }
        __syncthreads();
        const uint32_t tot = so[take], call = s_call;
        // entry i of the piece: the last tile whose entries start at or before it
#pragma unroll 4
        for (uint32_t i = tid; i < tot; i += kResThreads) {
            uint32_t q = 0;
#pragma unroll
            for (uint32_t b = kResThreads / 2; b; b >>= 1)
                if (q + b < take && so[q + b] <= i) q += b;
            su[i + i / kResEach] = a.unc[(size_t)(t0 + q) * kTileUnc + (i - so[q])].x + cbase + sc[q];
        }
        __syncthreads();
        int d[kResEach];  // accepted iff d >= a
#pragma unroll
        for (int e = 0; e < kResEach; e++) {
            const uint32_t k = tid * kResEach + e;
            d[e] = k < tot ? top - (int)su[k + tid] : INT32_MIN;
        }
        uint32_t start = abase + tid * kResEach / 2, mask = 0;
        for (int pass = 0; pass <= kResThreads; pass++) {  // thread k is settled after pass k at the latest
            int acc = (int)start;
            mask = 0;
#pragma unroll
            for (int e = 0; e < kResEach; e++)
                if (d[e] >= acc) {
                    mask |= 1u << e;
                    acc++;
                }
            uint32_t all;
            const uint32_t next = abase + block_excl_sum((uint32_t)(acc - (int)start), red, all);
            const bool moved = next != start;
            start = next;
            if (tid == kResThreads - 1) sbef[kResThreads] = abase + all;
            if (!__syncthreads_or(moved)) break;
        }
        smask[tid] = mask;
        sbef[tid] = start;
        {
            const uint32_t hi = __shfl_down_sync(0xffffffffu, mask, 1);
            if (!(tid & 1)) a.ok[words + tid / 2] = mask | (hi << 16);
        }
        __syncthreads();
        // uncertain acceptances before entry k of the piece
        const auto before = [&](uint32_t k) {
            const uint32_t r = k % kResEach;
            return sbef[k / kResEach] + (r ? (uint32_t)__popc(smask[k / kResEach] & ((1u << r) - 1u)) : 0u);
        };
        if (tid < take) {
            const uint32_t b = before(so[tid]);
            const uint32_t rank = s.i + cbase + sc[tid] + b;
            a.base[t] = rank;
            a.uoff[t] = words * 32 + so[tid];
            if (rank + c + (before(so[tid + 1]) - b) >= a.n) atomicMin(&s_end, t);
        }
        __syncthreads();
        t_end = s_end;
        cbase += call;
        abase = sbef[kResThreads];
        t0 += take;
        words += kPieceUnc / 32;
        __syncthreads();
    }
    if (tid) return;
    FyState z = s;
    if (t_end == 0xffffffffu) {
        z.pos += nt;
        z.i += cbase + abase;
        *a.seg = FySeg{nt, s.m};
    } else {
        // The permutation ends in tile t_end. gen_perm refills when its index
        // reaches the end of a buffer, the last accepted draw included: when
        // that draw is the buffer's last one, one more buffer is used. The
        // last acceptance has v = 0 (T = 0), so it is the buffer's last draw
        // iff that draw is 0 and was accepted (a 0 is always a candidate, so
        // it is the last candidate of the tile's last run).
        const unsigned long long te = s.pos + t_end;
        unsigned long long next = te / a.tpb + 1;
        if (te % a.tpb == a.tpb - 1 &&
            a.raw[((size_t)(te % a.ring_tiles) + 1) * (kRuns * a.rl * kListDraws) - 1] == 0) {
            const FyRun r = a.run[(size_t)t_end * kRuns + kRuns - 1];
            bool ok = true;
            if (r.unc && a.unc[(size_t)t_end * kTileUnc + r.upre + r.unc - 1].y == r.cnt - 1) {
                const uint32_t k = a.uoff[t_end] + r.upre + r.unc - 1;
                ok = (a.ok[k >> 5] >> (k & 31u)) & 1u;
            }
            if (ok) next++;
        }
        z.start = next;
        z.pos = next * a.tpb;
        z.i = 0;
        z.m++;
        z.done = z.m >= a.count;
        *a.seg = FySeg{t_end + 1, s.m};
    }
    // `bad` is only ever set, by this step's classification before this
    // launch or the emission after it
    a.state->pos = z.pos;
    a.state->start = z.start;
    a.state->m = z.m;
    a.state->i = z.i;
    a.state->done = z.done;
}

// Writes a step's accepted offsets at their ranks: a run's candidates without
// its rejected uncertain draws, which are marked in a bitmap so that ranks are
// popcounts. Checks that T at the start of every run lay in the window its
// classification assumed, which makes the whole step exact.
__global__ void __launch_bounds__(kRuns * 32, 4) k_fy_emit(FyScanArgs a) {
    constexpr uint32_t kWords = kMaxRunLists * kListDraws / 32;
    __shared__ uint32_t sacc[kRuns], bm[kRuns][kWords];
    const FySeg seg = *a.seg;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    uint32_t* acc = a.acc + ((size_t)seg.m * 3 + a.g) * a.n;
    for (uint32_t t = blockIdx.x; t < seg.ntiles; t += gridDim.x) {
        const FyRun r = a.run[(size_t)t * kRuns + w];
        const uint2* un = a.unc + (size_t)t * kTileUnc + r.upre;
        const uint32_t k0 = a.uoff[t] + r.upre;
        for (uint32_t j = lane; j * 32 < r.cnt; j += 32) bm[w][j] = 0;
        __syncwarp();
        uint32_t mine = 0;
        for (uint32_t j = lane; j < r.unc; j += 32) {
            const uint32_t p = un[j].y;
            const bool ok = (a.ok[(k0 + j) >> 5] >> ((k0 + j) & 31u)) & 1u;
            mine += ok;
            if (!ok && p < r.cnt) atomicOr(&bm[w][p >> 5], 1u << (p & 31u));
        }
        mine = __reduce_add_sync(0xffffffffu, mine);
        if (lane == 0) sacc[w] = mine;
        __syncthreads();
        uint32_t out = a.base[t] + r.cpre;
        for (int k = 0; k < w; k++) out += sacc[k];
        __syncthreads();
        const long long T = (long long)a.n - 1 - out;
        // past the permutation's end (T < 0) nothing may be certain
        const bool good = T >= 0 ? (T >= r.lo && T <= r.hi) : r.cnt == r.unc;
        if (!good && lane == 0) atomicOr(&a.state->bad, kMissed);
        const uint32_t* cand = a.cand + ((size_t)t * kRuns + w) * (a.rl * kListDraws);
        for (uint32_t b = 0; b < r.cnt; b += 256) {
            uint32_t v[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const uint32_t p = b + 32 * k + lane;
                v[k] = p < r.cnt ? cand[p] : 0u;
            }
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const uint32_t p = b + 32 * k + lane;
                if (b + 32 * k >= r.cnt) break;
                const uint32_t rej = bm[w][(b >> 5) + k];
                const uint32_t o = out + (lane - __popc(rej & lt));
                if (p < r.cnt && !((rej >> lane) & 1u) && o < a.n) acc[o] = v[k];
                out += 32 - __popc(rej);
            }
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// Small permutations (M = 2^bit_width(n) up to 2^16). A permutation then takes
// d ≈ M·H_n draws (std ≈ 1.3·M) and 1 + floor(d / 2^20) getNext buffers, a
// count that is predictable: permutation m of a group is assumed to start at
// buffer m·b̂ of the chain, and every (permutation, group) pair runs at once,
// one CTA each, with no host round trip. The CTA generates 8192 draws into
// shared memory and replays the acceptance on them min(8192, M) at a time: a
// thread holds consecutive draws and decides them from an assumed number of
// acceptances before its first, the block's prefix sums give the next
// assumption, until nothing changes (thread 0 starts from the true count; a
// threshold moves little over M draws, so a few passes do). A warp that walked
// the draws beside the generating warps was the bottleneck: 42 permutations of
// 20000 rows 1.77 and 0.93 ms, of 10000 rows 1.29 and 0.58, of 1000 rows 0.70
// and 0.21. The CTA reports the buffers used. The host then checks the assumed starts
// against the used counts; from the first permutation of a group whose start
// was wrong, the rest are run again from the corrected start (each pass
// fixes at least that one). A permutation needing more than `max_chunks`
// chunks sets `overflow`, and the pass is run again with twice as many (the
// chain below cannot take these: a run of it holds 2048 draws, of which more
// than kRunUnc are uncertain when M is that small).
constexpr uint32_t kSmallChunk = 8192;  // draws per chunk
constexpr int kSmallThreads = 512;
// Up to M = 2^15 always, at 2^16 from 18 permutations on: one permutation then
// takes its SM 1.2 ms however few there are, and a prediction fails in one of
// 140 to 270, which costs another pass, where the chain takes 70 to 80 us for
// each in turn. 33000 rows, mean of 12 seeds, chain and this path: 8
// permutations 0.92 and 1.32 ms, 20 1.71 and 1.55, 42 3.11 and 1.90, 66 4.57
// and 2.86; 65535 rows: 1.08 and 1.49, 1.99 and 1.75, 3.62 and 2.72, 5.17 and
// 4.07. At 2^17 a pass takes twice as long and a prediction fails twice as often.
inline bool fy_small_path(uint64_t M, size_t count) { return M <= 1u << 15 || (M == 1u << 16 && count >= 18); }
constexpr uint32_t kChunksPerBuffer = (1u << 20) / kSmallChunk;  // 128
constexpr uint32_t kSmallChunkLimit = (1u << 31) / kSmallChunk;   // draws are counted in 32 bits
constexpr size_t kSmallSmem = (size_t)kAesSmemBytes + kSmallChunk * 4;
constexpr int kSmallEach = kSmallChunk / kSmallThreads;  // 16: draws a thread decides at most at once

struct FySmallArgs {
    StreamArg st[3];  // chain start of each group (buffer 0)
    uint32_t n, mask, count, max_chunks;
    uint32_t m0[3];        // per group, the first permutation to run
    const uint32_t* start;  // [3][count] assumed start buffer
    uint32_t* used;         // [3][count] buffers used
    uint32_t* acc;          // [count][3][n] accepted offsets v_i
    uint32_t* overflow;     // set when a permutation needs more than max_chunks
};

__global__ void __launch_bounds__(kSmallThreads, 1) k_fy_small(FySmallArgs a) {
    const uint32_t m = blockIdx.x / 3, g = blockIdx.x % 3;
    if (m < a.m0[g]) return;  // already verified (uniform per CTA)
    extern __shared__ __align__(16) uint32_t sm[];
    __shared__ uint32_t s_dlast;
    aes_stage_tables(sm);
    const AesSmem S(sm);
    uint32_t* buf = sm + kAesSmemBytes / 4;  // [kSmallChunk]
    __shared__ uint32_t red[33];
    __shared__ CtrPre pre[2];
    const AesRK& rk = a.st[g].rk;
    const unsigned long long nonce = a.st[g].nonce + 4ull * a.start[g * a.count + m];  // 4 nonces per buffer
    const uint32_t n = a.n, tid = threadIdx.x;
    uint32_t* acc = a.acc + ((size_t)m * 3 + g) * n;
    const uint32_t mbits = 32 - __clz(a.mask);
    // draws a thread takes at once: at most M for the block
    const uint32_t each = min((uint32_t)kSmallEach, max(1u, (1u << mbits) / kSmallThreads));
    uint32_t i = 0;  // accepted so far
    for (uint32_t k = 0; k < a.max_chunks && i < n; k++) {
        const unsigned long long blk0 = (unsigned long long)k * (kSmallChunk / 4);
        if (!(blk0 & 0xffffu)) {  // a new nonce (the barrier below it has freed pre)
            if (tid < 2) pre[tid] = ctr_pre(S, rk, nonce + (blk0 >> 16), tid);
            __syncthreads();
        }
        for (uint32_t b = tid; b < kSmallChunk / 4; b += kSmallThreads) {
            const uint4 ks = keystream_block_pre(S, rk, pre, 0, blk0 + b);
            reinterpret_cast<uint4*>(buf)[b] = make_uint4(ks.x & a.mask, ks.y & a.mask, ks.z & a.mask, ks.w & a.mask);
        }
        __syncthreads();
        for (uint32_t s0 = 0; s0 < kSmallChunk && i < n; s0 += each * kSmallThreads) {
            const uint32_t T = n - 1 - i;
            const uint32_t d0 = s0 + tid * each;  // this thread's first draw of the chunk
            uint32_t v[kSmallEach];
            bool any = false;
#pragma unroll
            for (int e = 0; e < kSmallEach; e += 4) {
                uint4 x = make_uint4(0x7fffffffu, 0x7fffffffu, 0x7fffffffu, 0x7fffffffu);
                if ((uint32_t)e + 4 <= each) {  // (each is a power of two)
                    x = *reinterpret_cast<const uint4*>(buf + d0 + e);
                } else if (e == 0) {
                    x.x = buf[d0];
                    if (each > 1) x.y = buf[d0 + 1];
                }
                v[e] = x.x;
                v[e + 1] = x.y;
                v[e + 2] = x.z;
                v[e + 3] = x.w;
                any = any || min(min(x.x, x.y), min(x.z, x.w)) <= T;
            }
            // T only decreases: a stretch without a draw <= T has no acceptance
            if (!__syncthreads_or(any)) continue;
            uint32_t before = (uint32_t)(((unsigned long long)tid * each * (T + 1)) >> mbits), got = 0, all = 0;
            for (int pass = 0; pass <= kSmallThreads; pass++) {  // thread k is settled after pass k at the latest
                uint32_t x = before;
                got = 0;
#pragma unroll
                for (int e = 0; e < kSmallEach; e++)
                    if (v[e] + x <= T) {
                        got |= 1u << e;
                        x++;
                    }
                const uint32_t next = block_excl_sum(x - before, red, all);
                const bool moved = next != before;
                before = next;
                if (!__syncthreads_or(moved)) break;
            }
            uint32_t o = i + before;
#pragma unroll
            for (int e = 0; e < kSmallEach; e++)
                if ((got >> e) & 1u) {
                    acc[o] = v[e];  // o < n: an acceptance needs v + (acceptances before it) <= T
                    if (o == n - 1) s_dlast = k * kSmallChunk + d0 + e;
                    o++;
                }
            i += all;
        }
        __syncthreads();  // the next chunk rewrites the draws
    }
    if (tid == 0) {
        // gen_perm refills each time its index reaches the end of a buffer,
        // the last accepted draw included: 1 + floor(draws / 2^20) buffers
        if (i >= n) a.used[g * a.count + m] = 1u + (s_dlast + 1u) / (1u << 20);
        else atomicOr(a.overflow, 1u);
    }
}

// ---- finalize: accepted offsets -> permutation -----------------------------
// Step i swaps positions i and j_i = i + v_i (j_i >= i), so position i is final
// after step i. The steps s != k with j_s = k (all s < k) form the bucket of
// position k, s_1 < ... < s_c in step order. Position k holds k until step s_1
// and A(s_m) after step s_m, where A(s) is the value at position s just before
// step s. So step s_m outputs p[s_m] = A(s_{m-1}) (k for m = 1), and A(k) =
// A(s_c) (k for an empty bucket): A(k) is the root of k in the forest of links
// k -> max(bucket(k)). A self-swap (j_k = k) outputs p[k] = A(k).
// Buckets are built by a counting sort: counts per target, an exclusive scan
// per permutation, then an atomic cursor per target places the steps (the
// cursor ends at the bucket's end, which is also the next bucket's start).
constexpr int kFinThreads = 1024;
constexpr uint32_t kFinChunk = kFinThreads * 8;  // scan chunk
// Positions finalized at once: the random accesses of a batch's five arrays
// then stay in L2. 44 permutations of 2^22 rows (three groups): 111 ms with
// batches of 12 local permutations, 98 with 6, 87 with 2; smaller sizes take
// more per batch, down to one batch for all.
constexpr size_t kFinBatch = (size_t)1 << 23;

struct FinArgs {
    const uint32_t* acc;  // [P][n]
    uint32_t n, P, chunks;
    uint32_t* cur;        // [P][n] bucket sizes, then starts (scan), then ends (place)
    uint32_t* part;       // [P][chunks] chunk sums, then their exclusive scan
    int32_t* bucket;      // [P][n] steps grouped by target
    int32_t* par;         // [P][n] max(bucket(k)), -1 when empty
    int32_t* A;           // [P][n]
    int32_t* const* inv_out;   // [P] -> n
    int* err;
};

// target of step i; an out-of-range offset (never produced by a correct scan)
// is flagged and treated as a self-swap so no access leaves the arrays
__device__ __forceinline__ uint32_t fin_target(const FinArgs& a, size_t t, uint32_t i) {
    const unsigned long long j = (unsigned long long)i + a.acc[t];
    if (j >= a.n) {
        atomicOr(a.err, 1);
        return i;
    }
    return (uint32_t)j;
}

__global__ void k_fin_count(FinArgs a) {
    const size_t tot = (size_t)a.P * a.n;
    for (size_t t = gtid(); t < tot; t += gstride()) {
        const size_t pm = t / a.n;
        const uint32_t i = (uint32_t)(t % a.n);
        const uint32_t j = fin_target(a, t, i);
        if (j != i) atomicAdd(&a.cur[pm * a.n + j], 1u);
    }
}

// sum of chunk (blockIdx.x % chunks) of permutation (blockIdx.x / chunks)
__global__ void __launch_bounds__(kFinThreads) k_fin_part(FinArgs a) {
    __shared__ uint32_t red[33];
    const size_t pm = blockIdx.x / a.chunks, ch = blockIdx.x % a.chunks;
    const uint32_t* c = a.cur + pm * a.n;
    uint32_t s = 0;
#pragma unroll
    for (int u = 0; u < 8; u++) {
        const size_t k = ch * kFinChunk + (size_t)u * kFinThreads + threadIdx.x;
        s += k < a.n ? c[k] : 0u;
    }
    uint32_t tot;
    block_excl_sum(s, red, tot);
    if (threadIdx.x == 0) a.part[pm * a.chunks + ch] = tot;
}

// exclusive scan of one permutation's chunk sums (one CTA per permutation)
__global__ void __launch_bounds__(kFinThreads) k_fin_top(FinArgs a) {
    __shared__ uint32_t red[33];
    uint32_t* p = a.part + (size_t)blockIdx.x * a.chunks;
    uint32_t carry = 0;
    for (uint32_t b0 = 0; b0 < a.chunks; b0 += kFinThreads) {
        const uint32_t k = b0 + threadIdx.x;
        const uint32_t v = k < a.chunks ? p[k] : 0u;
        uint32_t tot;
        const uint32_t pre = block_excl_sum(v, red, tot);
        if (k < a.chunks) p[k] = carry + pre;
        carry += tot;
    }
}

// bucket starts: exclusive scan of the sizes, in place
__global__ void __launch_bounds__(kFinThreads) k_fin_starts(FinArgs a) {
    __shared__ uint32_t red[33];
    const size_t pm = blockIdx.x / a.chunks, ch = blockIdx.x % a.chunks;
    uint32_t* c = a.cur + pm * a.n;
    // coalesced: element u * kFinThreads + thread of the chunk, through shared
    // memory to 8 consecutive ones a thread for the scan and back (a thread's 8
    // consecutive global words took 47 us for 2^23 positions, now 16)
    __shared__ uint32_t sv[kFinChunk + kFinChunk / 8];
    const size_t c0 = ch * kFinChunk;
#pragma unroll
    for (int u = 0; u < 8; u++) {
        const uint32_t k = u * kFinThreads + threadIdx.x;
        sv[k + k / 8] = c0 + k < a.n ? c[c0 + k] : 0u;
    }
    __syncthreads();
    uint32_t v[8], s = 0;
#pragma unroll
    for (int u = 0; u < 8; u++) {
        v[u] = sv[threadIdx.x * 9 + u];
        s += v[u];
    }
    uint32_t tot;
    uint32_t pre = block_excl_sum(s, red, tot) + a.part[pm * a.chunks + ch];
#pragma unroll
    for (int u = 0; u < 8; u++) {
        sv[threadIdx.x * 9 + u] = pre;
        pre += v[u];
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 8; u++) {
        const uint32_t k = u * kFinThreads + threadIdx.x;
        if (c0 + k < a.n) c[c0 + k] = sv[k + k / 8];
    }
}

__global__ void k_fin_place(FinArgs a) {
    const size_t tot = (size_t)a.P * a.n;
    for (size_t t = gtid(); t < tot; t += gstride()) {
        const size_t pm = t / a.n;
        const uint32_t i = (uint32_t)(t % a.n);
        const uint32_t j = fin_target(a, t, i);
        if (j != i) {
            const uint32_t slot = atomicAdd(&a.cur[pm * a.n + j], 1u);
            if (slot < a.n) a.bucket[pm * a.n + slot] = (int32_t)i;
            else atomicOr(a.err, 2);
        }
    }
}

// bucket of position k after placement: [end(k-1), end(k)), clamped to n
__device__ __forceinline__ void fin_bucket(const FinArgs& a, size_t pm, uint32_t k, uint32_t& b, uint32_t& e) {
    const uint32_t* cur = a.cur + pm * a.n;
    e = min(cur[k], a.n);
    b = k ? min(cur[k - 1], e) : 0u;
}

__global__ void k_fin_par(FinArgs a) {
    const size_t tot = (size_t)a.P * a.n;
    for (size_t t = gtid(); t < tot; t += gstride()) {
        const size_t pm = t / a.n;
        const uint32_t k = (uint32_t)(t % a.n);
        uint32_t b, e;
        fin_bucket(a, pm, k, b, e);
        const int32_t* bk = a.bucket + pm * a.n;
        int32_t mx = -1;
        for (uint32_t m = b; m < e; m++) mx = max(mx, bk[m]);
        // bucket entries are steps before k; anything else is corruption
        if (mx >= (int32_t)k) {
            atomicOr(a.err, 8);
            mx = -1;
        }
        a.par[t] = mx;
    }
}

__global__ void k_fin_roots(FinArgs a) {
    const size_t tot = (size_t)a.P * a.n;
    for (size_t t = gtid(); t < tot; t += gstride()) {
        const size_t pm = t / a.n;
        const int32_t* par = a.par + pm * a.n;
        int32_t k = (int32_t)(t % a.n);
        int32_t p = par[k];
        while (p >= 0) {  // strictly decreasing links: ends at a root
            k = p;
            p = par[k];
        }
        a.A[t] = k;
    }
}

__device__ __forceinline__ void fin_emit(const FinArgs& a, size_t pm, uint32_t s, int32_t val) {
    if ((uint32_t)val >= a.n) {
        atomicOr(a.err, 4);
        val = (int32_t)s;
    }
    a.inv_out[pm][val] = (int32_t)s;
}

// per position k: its own step if it is a self-swap, and every step of its
// bucket (predecessor found by a scan of the small bucket)
__global__ void k_fin_final(FinArgs a) {
    const size_t tot = (size_t)a.P * a.n;
    for (size_t t = gtid(); t < tot; t += gstride()) {
        const size_t pm = t / a.n;
        const uint32_t k = (uint32_t)(t % a.n);
        const int32_t* A = a.A + pm * a.n;
        if (fin_target(a, t, k) == k) fin_emit(a, pm, k, A[k]);
        uint32_t b, e;
        fin_bucket(a, pm, k, b, e);
        const int32_t* bk = a.bucket + pm * a.n;
        for (uint32_t m = b; m < e; m++) {
            const int32_t s = bk[m];
            int32_t pred = -1;
            for (uint32_t q = b; q < e; q++) {
                const int32_t x = bk[q];
                if (x < s && x > pred) pred = x;
            }
            fin_emit(a, pm, (uint32_t)s, pred >= 0 ? A[pred] : (int32_t)k);
        }
    }
}

}  // namespace

// ---------------------------------------------------------------------------
// Generate `count` sharded permutations of size n from the three 2-party group
// streams, in ORQ's order: permutation-major, groups {0,1},{0,2},{1,2}
// (generateBatch, hm_sharded_permutation_generator.h:178-194).
namespace {
FyRes& fy_res(Ctx& c) {
    FyRes& R = c.fy;
    if (R.ready) return R;
    // the scans' streams have the highest priority: their small CTAs are
    // dispatched before the next generator launch's
    int prio_lo = 0, prio_hi = 0;
    ORQ_CUDA_CHECK(cudaDeviceGetStreamPriorityRange(&prio_lo, &prio_hi));
    ORQ_CUDA_CHECK(cudaStreamCreateWithPriority(&R.gs, cudaStreamNonBlocking, prio_lo));
    for (int g = 0; g < 3; g++) ORQ_CUDA_CHECK(cudaStreamCreateWithPriority(&R.ss[g], cudaStreamNonBlocking, prio_hi));
    ORQ_CUDA_CHECK(cudaStreamCreateWithPriority(&R.fs, cudaStreamNonBlocking, prio_lo));
    ORQ_CUDA_CHECK(cudaEventCreateWithFlags(&R.ev_start, cudaEventDisableTiming));
    ORQ_CUDA_CHECK(cudaEventCreateWithFlags(&R.fin_done, cudaEventDisableTiming));
    for (int k = 0; k < kFyInFlight; k++)
        for (int g = 0; g < 3; g++) {
            ORQ_CUDA_CHECK(cudaEventCreateWithFlags(&R.gen_done[g][k], cudaEventDisableTiming));
            ORQ_CUDA_CHECK(cudaEventCreateWithFlags(&R.st_ev[g][k], cudaEventDisableTiming));
        }
    ORQ_CUDA_CHECK(cudaMallocHost(&R.hst, (size_t)kFyInFlight * 3 * sizeof(FyState)));
    R.ready = true;
    return R;
}
}  // namespace

void release_fy(Ctx& c) {
    FyRes& R = c.fy;
    if (!R.ready) return;
    cudaStreamSynchronize(R.gs);
    for (int g = 0; g < 3; g++) cudaStreamSynchronize(R.ss[g]);
    cudaStreamSynchronize(R.fs);
    cudaEventDestroy(R.ev_start);
    cudaEventDestroy(R.fin_done);
    for (int k = 0; k < kFyInFlight; k++)
        for (int g = 0; g < 3; g++) {
            cudaEventDestroy(R.gen_done[g][k]);
            cudaEventDestroy(R.st_ev[g][k]);
        }
    cudaStreamDestroy(R.gs);
    for (int g = 0; g < 3; g++) cudaStreamDestroy(R.ss[g]);
    cudaStreamDestroy(R.fs);
    cudaFreeHost(R.hst);
    R = FyRes{};
}

namespace {
// How `count` permutations of n > 0 rows are generated on num_sms SMs.
struct FyPlan {
    int bitsw;               // M = 2^bitsw
    double M, H, per_perm;   // harmonic number of n, expected getNext buffers
    bool small;
    size_t fin_p;            // local permutations finalized at once
    uint32_t fin_chunks;     // scan chunks of a permutation
    // the chain
    uint32_t gen_sms, W, rl, tpb, ring_bufs, ring_tiles, seg_cap;
};
FyPlan fy_plan(int num_sms, size_t n, size_t count) {
    FyPlan p{};
    while (p.bitsw < 64 && (n >> p.bitsw)) p.bitsw++;
    p.M = (double)(1ull << p.bitsw);
    for (size_t k = 1; k <= std::min<size_t>(n, 1 << 16); k++) p.H += 1.0 / k;
    if (n > (1u << 16)) p.H += std::log((double)n / (1 << 16));
    p.per_perm = p.M * p.H / (double)(1 << 20) + 1.0;
    p.small = fy_small_path(1ull << p.bitsw, count);
    p.fin_p = std::clamp<size_t>(kFinBatch / n, 1, 3 * count);
    p.fin_chunks = (uint32_t)ceil_div(n, (size_t)kFinChunk);
    // Buffers are generated `W` at a time per group into a ring of kRing * W
    // (up to kRing - 1 chunks ahead of the scan: the draws do not depend on
    // it). W buffers of 2^20 draws keep every SM busy for ~6 us each.
    constexpr uint32_t kRing = 4;
    // Three SMs are left to k_fy_resolve, whose registers do not fit beside a
    // generator CTA's; up to M = 2^19, where the chain waits for its steps and
    // not for the generator, 24 (44 permutations of 100003 rows 4.8 and 4.0 ms,
    // of 262143 7.4 and 6.4; of 2^19 rows, M = 2^20, 11.6 and 11.4). W is
    // rounded so that the last wave of lists is full.
    p.gen_sms = (uint32_t)std::max(1, num_sms - (p.bitsw <= 19 ? std::min(24, num_sms / 6) : 3));
    const uint32_t gen_warps = p.gen_sms * (kGenThreads / 32);
    const double want = std::clamp(p.per_perm * count / 8.0, 2.0, 64.0);
    const uint32_t waves = std::max(1u, (uint32_t)(want * kListsPerBuf / gen_warps));
    p.W = std::max(2u, waves * gen_warps / kListsPerBuf);
    // Runs of 8192 draws, or shorter ones where a permutation has few of them:
    // a step's latency is then what counts, and more warps share its draws.
    p.rl = p.M >= (double)(1u << 22) ? 4 : (p.M >= (double)(1u << 20) ? 2 : 1);
    p.tpb = kListsPerBuf / (kRuns * p.rl);
    p.ring_bufs = kRing * p.W;
    p.ring_tiles = p.ring_bufs * p.tpb;
    p.seg_cap = p.W * p.tpb;
    return p;
}

// The buffers of one group's chain.
enum { RING_RAW, RING_LST, RING_LCNT, RING_TAB, RING_CAND, RING_UNC, RING_RUN, RING_TC, RING_TU, RING_BASE, RING_UOFF, RING_OK, RING_N };
void ring_bytes(const FyPlan& p, size_t (&b)[RING_N]) {
    b[RING_RAW] = (size_t)p.ring_bufs * kBufDraws * 4;
    b[RING_LST] = (size_t)p.ring_bufs * kListsPerBuf * kListCap * 4;
    b[RING_LCNT] = (size_t)p.ring_bufs * kListsPerBuf * 4;
    b[RING_TAB] = (size_t)p.ring_bufs * 4 * kTabEntries * sizeof(uint4);
    b[RING_CAND] = (size_t)p.W * kBufDraws * 4;
    b[RING_UNC] = (size_t)p.seg_cap * kTileUnc * sizeof(uint2);
    b[RING_RUN] = (size_t)p.seg_cap * kRuns * sizeof(FyRun);
    b[RING_TC] = b[RING_TU] = b[RING_BASE] = b[RING_UOFF] = (size_t)p.seg_cap * 4;
    b[RING_OK] = (size_t)p.seg_cap * (kPieceUnc / 8);  // (a piece of k_fy_resolve takes at least one tile)
}
}  // namespace

size_t perm_bytes(int num_sms, size_t n, size_t count) {
    if (!count) return 0;
    size_t t = count * pool_block(3 * std::max<size_t>(n, 1) * 4);
    if (!n) return t;
    const FyPlan p = fy_plan(num_sms, n, count);
    const size_t el = p.fin_p * n;
    t += pool_block(3 * count * n * 4) + 4 * pool_block(el * 4) + pool_block(p.fin_p * p.fin_chunks * 4) +
         pool_block(3 * count * sizeof(void*));
    if (p.small) return t + 2 * pool_block(3 * count * 4) + pool_block(4);
    size_t b[RING_N];
    ring_bytes(p, b);
    for (size_t x : b) t += 3 * pool_block(x);
    return t + pool_block(3 * sizeof(FyState)) + pool_block(3 * sizeof(FySeg));
}

void gen_sharded_perms(Ctx& c, size_t n, size_t count, std::vector<ShardedPerm>& out) {
    out.clear();
    if (count == 0) return;
    if (n >= (1ull << 31)) throw std::invalid_argument("permutation size must be < 2^31");
    out.resize(count);
    for (auto& sp : out) {
        sp.n = n;
        int32_t* inv = (int32_t*)c.alloc(3 * std::max<size_t>(n, 1) * 4);
        for (int g = 0; g < 3; g++) sp.inv[g] = inv + g * n;
    }
    if (n == 0) {
        // gen_perm still draws one buffer (4 nonces) per permutation
        for (int g = 0; g < 3; g++) c.nonce[G01 + g] += 4ull * count;
        return;
    }
    const FyPlan plan = fy_plan(c.num_sms, n, count);
    const double M = plan.M, H = plan.H, per_perm = plan.per_perm;
    const uint32_t mask = (uint32_t)((1ull << plan.bitsw) - 1);
    Scratch acc(c, (size_t)3 * count * n * 4);
    // generator and scans run on private non-blocking streams so they overlap
    // whatever the caller's stream is (the legacy default stream included)
    FyRes& R = fy_res(c);
    cudaStream_t gs = R.gs;
    cudaStream_t* ss = R.ss;
    cudaEvent_t ev_start = R.ev_start;
    // On every exit path (an exception included) the generator and scanner
    // streams are drained before the ring, state and output scratch above go
    // back to the pool: a later call on the runtime's stream could otherwise
    // be handed memory those kernels are still writing. Declared after the
    // scratch buffers, so it runs before their destructors.
    //
    // Finalize runs on its own low-priority stream for the permutations the
    // scanners have completed, while the chain goes on (the generator leaves
    // SMs idle while the scanners work through dense windows). acc is laid out
    // [permutation][group], so consecutive local permutations are one
    // contiguous batch; the scratch holds one batch.
    const size_t fin_p = plan.fin_p, fin_el = fin_p * n;
    const uint32_t fin_chunks = plan.fin_chunks;
    Scratch f_cur(c, fin_el * 4), f_part(c, fin_p * fin_chunks * 4), f_bucket(c, fin_el * 4),
        f_par(c, fin_el * 4), f_A(c, fin_el * 4), f_ptrs(c, 3 * count * sizeof(void*));
    {
        std::vector<int32_t*> hp(3 * count);
        for (size_t m = 0; m < count; m++)
            for (int g = 0; g < 3; g++) hp[3 * m + g] = out[m].inv[g];
        ORQ_CUDA_CHECK(cudaMemcpyAsync(f_ptrs.p, hp.data(), hp.size() * sizeof(void*), cudaMemcpyHostToDevice,
                                       c.stream));
        ORQ_CUDA_CHECK(cudaStreamSynchronize(c.stream));  // hp is pageable and leaves scope
    }
    cudaStream_t fs = R.fs;
    size_t fin_next = 0;  // local permutations [0, fin_next) are queued for finalize
    auto launch_fin = [&](size_t q0, size_t q1) {
        const size_t P = q1 - q0;
        const size_t el = P * n;
        FinArgs fa;
        fa.acc = acc.as<uint32_t>() + q0 * n;
        fa.n = (uint32_t)n;
        fa.P = (uint32_t)P;
        fa.chunks = fin_chunks;
        fa.cur = f_cur.as<uint32_t>();
        fa.part = f_part.as<uint32_t>();
        fa.bucket = f_bucket.as<int32_t>();
        fa.par = f_par.as<int32_t>();
        fa.A = f_A.as<int32_t>();
        fa.inv_out = f_ptrs.as<int32_t*>() + q0;
        fa.err = c.d_err;
        const unsigned gg = plain_grid(c, el);
        const unsigned gc = (unsigned)(P * fin_chunks);
        ProfScope ps(c, "fy_finalize", 0.0, 0.0, fs);
        ORQ_CUDA_CHECK(cudaMemsetAsync(f_cur.p, 0, el * 4, fs));
        k_fin_count<<<gg, 256, 0, fs>>>(fa);
        k_fin_part<<<gc, kFinThreads, 0, fs>>>(fa);
        k_fin_top<<<(unsigned)P, kFinThreads, 0, fs>>>(fa);
        k_fin_starts<<<gc, kFinThreads, 0, fs>>>(fa);
        k_fin_place<<<gg, 256, 0, fs>>>(fa);
        k_fin_par<<<gg, 256, 0, fs>>>(fa);
        k_fin_roots<<<gg, 256, 0, fs>>>(fa);
        k_fin_final<<<gg, 256, 0, fs>>>(fa);
        ORQ_CUDA_CHECK(cudaGetLastError());
        c.kernels_launched += 8;
    };
    struct DrainSideStreams {
        FyRes& r;
        ~DrainSideStreams() {
            cudaStreamSynchronize(r.gs);
            for (int g = 0; g < 3; g++) cudaStreamSynchronize(r.ss[g]);
            cudaStreamSynchronize(r.fs);
        }
    } drain{R};
    ORQ_CUDA_CHECK(cudaEventRecord(ev_start, c.stream));
    ORQ_CUDA_CHECK(cudaStreamWaitEvent(gs, ev_start, 0));
    for (int g = 0; g < 3; g++) ORQ_CUDA_CHECK(cudaStreamWaitEvent(ss[g], ev_start, 0));
    ORQ_CUDA_CHECK(cudaStreamWaitEvent(fs, ev_start, 0));

    if (plan.small) {
        // every permutation of every group at once from predicted start
        // buffers, corrected pass by pass (k_fy_small)
        const uint32_t bhat = (uint32_t)std::max(1, 1 + (int)(M * H / (double)(1u << 20)) + c.fy_tune.buffers);
        std::vector<uint32_t> hstart(3 * count), hused(3 * count);
        for (int g = 0; g < 3; g++)
            for (size_t m = 0; m < count; m++) hstart[g * count + m] = (uint32_t)m * bhat;
        Scratch d_start(c, hstart.size() * 4), d_used(c, hused.size() * 4), ovf(c, 4);
        // the pool hands out memory in the runtime stream's order
        ORQ_CUDA_CHECK(cudaEventRecord(ev_start, c.stream));
        ORQ_CUDA_CHECK(cudaStreamWaitEvent(gs, ev_start, 0));
        ORQ_CUDA_CHECK(cudaMemsetAsync(ovf.p, 0, 4, gs));
        ORQ_CUDA_CHECK(cudaFuncSetAttribute(k_fy_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSmem));
        FySmallArgs sa;
        for (int g = 0; g < 3; g++) {
            sa.st[g] = c.stream_arg(G01 + g);
            sa.m0[g] = 0;
        }
        sa.n = (uint32_t)n;
        sa.mask = mask;
        sa.count = (uint32_t)count;
        sa.max_chunks = c.fy_tune.chunks ? c.fy_tune.chunks : (bhat + 6) * kChunksPerBuffer;
        sa.start = d_start.as<uint32_t>();
        sa.used = d_used.as<uint32_t>();
        sa.acc = acc.as<uint32_t>();
        sa.overflow = ovf.as<uint32_t>();
        for (bool again = true; again;) {
            ORQ_CUDA_CHECK(cudaMemcpyAsync(d_start.p, hstart.data(), hstart.size() * 4, cudaMemcpyHostToDevice, gs));
            {
                ProfScope ps(c, "fy_small", 0.0, 0.0, gs);
                k_fy_small<<<(unsigned)(3 * count), kSmallThreads, kSmallSmem, gs>>>(sa);
            }
            ORQ_CUDA_CHECK(cudaGetLastError());
            c.kernels_launched++;
            uint32_t overflow = 0;
            ORQ_CUDA_CHECK(cudaMemcpyAsync(hused.data(), d_used.p, hused.size() * 4, cudaMemcpyDeviceToHost, gs));
            ORQ_CUDA_CHECK(cudaMemcpyAsync(&overflow, ovf.p, 4, cudaMemcpyDeviceToHost, gs));
            ORQ_CUDA_CHECK(cudaStreamSynchronize(gs));
            if (overflow) {
                // the same pass with room for more draws (some `used` are not set)
                if (sa.max_chunks > kSmallChunkLimit / 2)
                    throw std::runtime_error("permutation generation did not converge");
                sa.max_chunks *= 2;
                ORQ_CUDA_CHECK(cudaMemsetAsync(ovf.p, 0, 4, gs));
                continue;
            }
            // permutations before m0[g] are verified, and so is m0[g]'s start;
            // the first one whose assumed start differs from the true one is
            // where the next pass begins (so every pass verifies at least one)
            again = false;
            for (int g = 0; g < 3; g++) {
                uint32_t* st = hstart.data() + g * count;
                const uint32_t* us = hused.data() + g * count;
                size_t m = sa.m0[g];
                if (m >= count) continue;
                uint32_t expect = st[m];
                for (; m < count; m++) {
                    if (st[m] != expect) break;
                    expect = st[m] + us[m];
                }
                sa.m0[g] = (uint32_t)m;
                if (m < count) {
                    again = true;
                    for (size_t k = m; k < count; k++) st[k] = expect + (uint32_t)(k - m) * bhat;
                }
            }
        }
        for (int g = 0; g < 3; g++)
            c.nonce[G01 + g] += 4ull * (hstart[g * count + count - 1] + hused[g * count + count - 1]);
        for (; fin_next < 3 * count; fin_next += fin_p) launch_fin(fin_next, std::min(3 * count, fin_next + fin_p));
        ORQ_CUDA_CHECK(cudaEventRecord(R.fin_done, fs));
        ORQ_CUDA_CHECK(cudaStreamWaitEvent(c.stream, R.fin_done, 0));
        c.check_device_error();
        return;
    }

    const uint32_t W = plan.W, rl = plan.rl, tpb = plan.tpb, gen_sms = plan.gen_sms;
    const uint32_t ring_bufs = plan.ring_bufs, ring_tiles = plan.ring_tiles, seg_cap = plan.seg_cap;
    struct Group {
        std::unique_ptr<Scratch> buf[RING_N];
        unsigned long long gen = 0;   // buffers generated (or queued)
        unsigned long long pos = 0;   // tiles known to be scanned
        unsigned long long start = 0;
        uint32_t m = 0;
        bool done = false;
        unsigned head = 0, tail = 0;  // step batches queued / read back
    } G[3];
    size_t rb_bytes[RING_N];
    ring_bytes(plan, rb_bytes);
    for (auto& q : G)
        for (int k = 0; k < RING_N; k++) q.buf[k].reset(new Scratch(c, rb_bytes[k]));
    Scratch state(c, 3 * sizeof(FyState)), seg(c, 3 * sizeof(FySeg));
    ORQ_CUDA_CHECK(cudaMemsetAsync(state.p, 0, 3 * sizeof(FyState), c.stream));
    // the side streams start after these allocations and the memset, and are
    // drained before the buffers above go back to the pool (declared after them)
    ORQ_CUDA_CHECK(cudaEventRecord(ev_start, c.stream));
    ORQ_CUDA_CHECK(cudaStreamWaitEvent(gs, ev_start, 0));
    for (int g = 0; g < 3; g++) ORQ_CUDA_CHECK(cudaStreamWaitEvent(ss[g], ev_start, 0));
    DrainSideStreams drain_ring{R};
    prep_aes_kernel(k_fy_gen);
    FyState* hst = static_cast<FyState*>(R.hst);

    // runs the chain; what went wrong, if anything (kMissed, kOverflow)
    const auto run_chain = [&](double width) -> uint32_t {
    FyScanArgs sa[3];
    for (int g = 0; g < 3; g++) {
        FyScanArgs& x = sa[g];
        x.n = (uint32_t)n;
        x.count = (uint32_t)count;
        x.g = (uint32_t)g;
        x.mbits = (uint32_t)plan.bitsw;
        x.th = (uint32_t)(n >> 4);
        x.rl = rl;
        x.tpb = tpb;
        x.ring_tiles = ring_tiles;
        x.seg_cap = seg_cap;
        x.limit = 0;
        x.rate = std::log1p(-1.0 / M);
        x.width = width;
        x.raw = G[g].buf[RING_RAW]->as<uint32_t>();
        x.lst = G[g].buf[RING_LST]->as<uint32_t>();
        x.lcnt = G[g].buf[RING_LCNT]->as<uint32_t>();
        x.state = state.as<FyState>() + g;
        x.cand = G[g].buf[RING_CAND]->as<uint32_t>();
        x.unc = G[g].buf[RING_UNC]->as<uint2>();
        x.run = G[g].buf[RING_RUN]->as<FyRun>();
        x.tc = G[g].buf[RING_TC]->as<uint32_t>();
        x.tu = G[g].buf[RING_TU]->as<uint32_t>();
        x.base = G[g].buf[RING_BASE]->as<uint32_t>();
        x.uoff = G[g].buf[RING_UOFF]->as<uint32_t>();
        x.ok = G[g].buf[RING_OK]->as<uint32_t>();
        x.seg = seg.as<FySeg>() + g;
        x.acc = acc.as<uint32_t>();
    }
    // a step ends with its permutation: a batch of steps covers the
    // permutations a chunk of buffers can hold, and one step more
    const int steps = (int)(W / per_perm) + 2;
    const unsigned scan_grid = (unsigned)std::min<uint32_t>(seg_cap, (uint32_t)std::max(1, 2 * c.num_sms));
    const auto queue_steps = [&](int g) {
        Group& q = G[g];
        const unsigned k = q.head % kFyInFlight;
        for (int s = 0; s < steps; s++) {
            ProfScope ps(c, "fy_scan", 0.0, 0.0, ss[g]);
            k_fy_classify<<<scan_grid, kRuns * 32, 0, ss[g]>>>(sa[g]);
            k_fy_resolve<<<1, kResThreads, 0, ss[g]>>>(sa[g]);
            k_fy_emit<<<scan_grid, kRuns * 32, 0, ss[g]>>>(sa[g]);
            c.kernels_launched += 3;
        }
        ORQ_CUDA_CHECK(cudaGetLastError());
        ORQ_CUDA_CHECK(cudaMemcpyAsync(hst + kFyInFlight * g + k, state.as<FyState>() + g, sizeof(FyState),
                                       cudaMemcpyDeviceToHost, ss[g]));
        ORQ_CUDA_CHECK(cudaEventRecord(R.st_ev[g][k], ss[g]));
        q.head++;
    };
    uint32_t bad = 0;
    // waits for the oldest batch of steps queued for g
    const auto read_back = [&](int g) {
        Group& q = G[g];
        if (q.head == q.tail) queue_steps(g);
        const unsigned k = q.tail++ % kFyInFlight;
        ORQ_CUDA_CHECK(cudaEventSynchronize(R.st_ev[g][k]));
        const FyState& z = hst[kFyInFlight * g + k];
        q.pos = z.pos;
        q.start = z.start;
        q.m = z.m;
        q.done = z.done != 0;
        bad |= z.bad;
        const size_t mmin = std::min({G[0].m, G[1].m, G[2].m});
        // the accepted offsets of these permutations precede the states read
        if (!bad && mmin < count)
            for (; fin_next + fin_p <= 3 * mmin; fin_next += fin_p) launch_fin(fin_next, fin_next + fin_p);
    };
    // Chunks shrink once a chain may end (a permutation's draws deviate by
    // ~1.3 M), and then each waits for the scan of the one before it, so that
    // little is generated past the end.
    const double sure = per_perm * count - 2.6 * M * std::sqrt((double)count) / kBufDraws;
    const double far = per_perm * 4.0 * count + 64.0 * count + 64.0;
    while (!bad) {
        int g = -1;
        for (int k = 0; k < 3; k++)
            if (!G[k].done && (g < 0 || G[k].gen < G[g].gen)) g = k;
        if (g < 0) break;
        Group& q = G[g];
        if ((double)q.gen > far) throw std::runtime_error("permutation generation did not converge");
        const bool tail = (double)q.gen >= sure;
        unsigned long long b = q.gen;
        // the chain never reads buffers before the current permutation's start
        uint32_t take = tail ? std::max(1u, W / 4) : W;
        take = (uint32_t)std::min<unsigned long long>(take, ring_bufs - b % ring_bufs);
        // wait until the ring slots are free, and in the tail for every scan
        if (q.head - q.tail == kFyInFlight || (b + take) * tpb > q.pos + ring_tiles ||
            (tail && q.head != q.tail)) {
            read_back(g);
            continue;
        }
        if (tail && q.pos < b * tpb) {  // the queued steps stopped short of what is generated
            read_back(g);
            continue;
        }
        const size_t rb = b % ring_bufs;
        uint4* tab = G[g].buf[RING_TAB]->as<uint4>() + rb * 4 * kTabEntries;
        FyGenArgs ga;
        ga.st = c.stream_arg(G01 + g, 4ull * b);
        ga.tab = tab;
        ga.mask = mask;
        ga.th = (uint32_t)(n >> 4);
        ga.lists = take * kListsPerBuf;
        ga.raw = G[g].buf[RING_RAW]->as<uint32_t>() + rb * kBufDraws;
        ga.lst = G[g].buf[RING_LST]->as<uint32_t>() + rb * kListsPerBuf * kListCap;
        ga.lcnt = G[g].buf[RING_LCNT]->as<uint32_t>() + rb * kListsPerBuf;
        ga.state = state.as<FyState>() + g;
        {
            ProfScope ps(c, "fy_gen", 0.0, (double)take * kBufDraws / 4, gs);
            k_fy_tab<<<take * 4, 544, 0, gs>>>(ga.st, tab);
            k_fy_gen<<<gen_sms, kGenThreads, kAesSmemBytes, gs>>>(ga);
        }
        ORQ_CUDA_CHECK(cudaGetLastError());
        c.kernels_launched += 2;
        q.gen = b + take;
        sa[g].limit = q.gen * tpb;
        ORQ_CUDA_CHECK(cudaEventRecord(R.gen_done[g][q.head % kFyInFlight], gs));
        ORQ_CUDA_CHECK(cudaStreamWaitEvent(ss[g], R.gen_done[g][q.head % kFyInFlight], 0));
        queue_steps(g);
    }
    // the last steps' emissions may still flag a window
    for (int g = 0; g < 3; g++) ORQ_CUDA_CHECK(cudaStreamSynchronize(ss[g]));
    ORQ_CUDA_CHECK(cudaMemcpyAsync(hst, state.p, 3 * sizeof(FyState), cudaMemcpyDeviceToHost, gs));
    ORQ_CUDA_CHECK(cudaStreamSynchronize(gs));
    for (int g = 0; g < 3; g++) {
        bad |= hst[g].bad;
        G[g].start = hst[g].start;
    }
    return bad;
    };
    // A threshold outside its window (6 deviations: about once in 1e7
    // permutations) shows up as kMissed: nothing has been consumed yet, so the
    // chain runs again with wider windows. Windows so wide that a run's
    // uncertain draws overflow (a quarter of M, some 80 deviations at M = 2^16)
    // are narrowed instead.
    double width = c.fy_tune.width;
    for (int tries = 1; const uint32_t bad = run_chain(width); tries++) {
        if (tries == 24) throw std::runtime_error("permutation generation did not converge");
        width *= bad & kOverflow ? 0.6 : 1.5;
        ORQ_CUDA_CHECK(cudaStreamSynchronize(fs));
        ORQ_CUDA_CHECK(cudaMemsetAsync(state.p, 0, 3 * sizeof(FyState), gs));
        ORQ_CUDA_CHECK(cudaStreamSynchronize(gs));
        for (auto& q : G) {
            q.gen = q.pos = q.start = 0;
            q.m = 0;
            q.done = false;
            q.head = q.tail = 0;
        }
    }
    // nonce accounting: 4 nonces per getNext buffer
    for (int g = 0; g < 3; g++) c.nonce[G01 + g] += 4ull * G[g].start;

    // the permutations completed since the last batch, then the runtime's
    // stream waits for the finalize stream
    for (; fin_next < 3 * count; fin_next += fin_p) launch_fin(fin_next, std::min(3 * count, fin_next + fin_p));
    ORQ_CUDA_CHECK(cudaEventRecord(R.fin_done, fs));
    ORQ_CUDA_CHECK(cudaStreamWaitEvent(c.stream, R.fin_done, 0));
    c.check_device_error();

}

namespace {
__global__ void k_invert(const int32_t* inv, int32_t* perm, unsigned long long n, int* err) {
    for (unsigned long long v = gtid(); v < n; v += gstride()) {
        const uint32_t s = (uint32_t)inv[v];
        if (s < n) perm[s] = (int32_t)v;
        else atomicOr(err, 4);
    }
}
}  // namespace

void ensure_perm(Ctx& c, ShardedPerm& sp) {
    if (sp.perm[0]) return;
    int32_t* p = (int32_t*)c.alloc(3 * std::max<size_t>(sp.n, 1) * 4);
    for (int g = 0; g < 3; g++) sp.perm[g] = p + g * sp.n;
    if (!sp.n) return;
    for (int g = 0; g < 3; g++) {
        k_invert<<<plain_grid(c, sp.n), 256, 0, c.stream>>>(sp.inv[g], sp.perm[g], sp.n, c.d_err);
        ORQ_CUDA_CHECK(cudaGetLastError());
        c.kernels_launched++;
    }
}

// PermutationManager::reserve (permutation_manager.h:102-181): keep a queue of
// permutations of one size; a size change empties it.
void reserve_perms(Ctx& c, size_t n, size_t count) {
    if (!c.perm_queue.empty() && c.perm_queue_n != n) {
        for (auto& sp : c.perm_queue) c.free_perm(sp);
        c.perm_queue.clear();
    }
    c.perm_queue_n = n;
    if (c.perm_queue.size() >= count) return;
    std::vector<ShardedPerm> fresh;
    gen_sharded_perms(c, n, count - c.perm_queue.size(), fresh);
    for (auto& sp : fresh) c.perm_queue.push_back(sp);
}

// PermutationManager::getNext / getNextPair for 3PC: pop the queue, or
// generate one on demand (hm generator getNext).
ShardedPerm next_perm(Ctx& c, size_t n) {
    if (!c.perm_queue.empty()) {
        if (c.perm_queue_n != n) throw std::runtime_error("queued permutation has the wrong size");
        ShardedPerm sp = c.perm_queue.front();
        c.perm_queue.pop_front();
        return sp;
    }
    std::vector<ShardedPerm> one;
    gen_sharded_perms(c, n, 1, one);
    return one[0];
}

}  // namespace orqcu
