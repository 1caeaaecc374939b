// aes.cuh — AES-256 keystream on sm_100a, laid out for ORQ's PRG.
//
// ORQ's AESPRGAlgorithm (include/core/random/prg/prg_algorithm.h:161-231) fills
// a buffer by AES-256-GCM-encrypting zeros in 1 MiB chunks; chunk c uses the
// 96-bit IV (nonce0 + c as 8 little-endian bytes, then 4 zero bytes) and, as
// GCM specifies (NIST SP 800-38D), block j of the chunk is
// AES_K(IV || BE32(j + 2)). Byte o of a stream draw is therefore keystream
// block (o >> 4) of chunk (o >> 20), an affine function of the element index:
// every thread can produce exactly the keystream its elements need.
//
// Implementation: the 32-bit "T-table" formulation of the AES round (FIPS-197
// §5.1 SubBytes+ShiftRows+MixColumns folded into four 256-entry tables).
// Tables live in shared memory replicated once per lane (entry x of table t
// for lane l at word  region(t)*16384 + x*64 + (t&1)*32 + l), so every lookup
// of a warp hits 32 distinct banks whatever the byte values are. The byte
// extraction and the lane offset fuse into one byte-permute: the lookup
// address is (byte << 8) | (lane << 2). Round keys come from kernel parameters
// (constant bank), so AddRoundKey costs no loads.
#pragma once
#include <cstdint>

namespace orqcu {

struct AesRK {
    uint32_t k[60];  // FIPS-197 key schedule, word i = key-schedule bytes 4i..4i+3 (LE)
};

// One PRG stream as a kernel sees it: key schedule + nonce of its first chunk.
struct StreamArg {
    AesRK rk;
    unsigned long long nonce;
};

constexpr int kAesSmemBytes = 2 * 256 * 256;  // 4 tables x 256 entries x 32 lanes x 4 B

// Global copy of T0..T3 (4 x 256 words). Each translation unit that launches
// AES kernels owns one copy (no device linking); common.cuh registers an
// uploader per unit and the runtime fills every copy once per device.
static __device__ uint32_t g_aes_T[4 * 256];

// The 32 lane copies of one entry are 128 contiguous bytes; a thread writes 4
// of them with one 128-bit store, so a quarter-warp store phase covers one
// 128-byte row (conflict-free) and each global word is read by 8 threads.
__device__ __forceinline__ void aes_stage_tables(uint32_t* sm) {
    constexpr int kStores = 4 * 256 * 8;
    for (int base = 0; base < kStores; base += 16 * blockDim.x) {
        uint32_t v[16];
#pragma unroll
        for (int u = 0; u < 16; u++) {
            const int idx = base + u * blockDim.x + threadIdx.x;
            v[u] = idx < kStores ? __ldg(&g_aes_T[idx >> 3]) : 0u;
        }
#pragma unroll
        for (int u = 0; u < 16; u++) {
            const int idx = base + u * blockDim.x + threadIdx.x;
            if (idx < kStores) {
                const int e = idx >> 3, t = e >> 8, x = e & 255;
                reinterpret_cast<uint4*>(sm + (t >> 1) * 16384 + x * 64 + (t & 1) * 32)[idx & 7] =
                    make_uint4(v[u], v[u], v[u], v[u]);
            }
        }
    }
    __syncthreads();
}

struct AesSmem {
    const char* base;  // shared base + lane*4 folded into the permute, see lk()
    uint32_t lane4;
    __device__ __forceinline__ explicit AesSmem(const uint32_t* sm)
        : base(reinterpret_cast<const char*>(sm)), lane4((threadIdx.x & 31u) << 2) {}
    // table t, byte j of word w
    template <int T, int J>
    __device__ __forceinline__ uint32_t lk(uint32_t w) const {
        const uint32_t a = __byte_perm(w, lane4, 0x5504u | (J << 4));
        return *reinterpret_cast<const uint32_t*>(base + a + (T >> 1) * 65536 + (T & 1) * 128);
    }
};

// One full round (1..13) in place.
__device__ __forceinline__ void aes256_round(const AesSmem& S, const AesRK& rk, const int r, uint32_t& s0, uint32_t& s1,
                                             uint32_t& s2, uint32_t& s3) {
    const uint32_t n0 = S.lk<0, 0>(s0) ^ S.lk<1, 1>(s1) ^ S.lk<2, 2>(s2) ^ S.lk<3, 3>(s3) ^ rk.k[4 * r + 0];
    const uint32_t n1 = S.lk<0, 0>(s1) ^ S.lk<1, 1>(s2) ^ S.lk<2, 2>(s3) ^ S.lk<3, 3>(s0) ^ rk.k[4 * r + 1];
    const uint32_t n2 = S.lk<0, 0>(s2) ^ S.lk<1, 1>(s3) ^ S.lk<2, 2>(s0) ^ S.lk<3, 3>(s1) ^ rk.k[4 * r + 2];
    const uint32_t n3 = S.lk<0, 0>(s3) ^ S.lk<1, 1>(s0) ^ S.lk<2, 2>(s1) ^ S.lk<3, 3>(s2) ^ rk.k[4 * r + 3];
    s0 = n0;
    s1 = n1;
    s2 = n2;
    s3 = n3;
}

// Rounds R0..14 of one block, in place, from the state after round R0 - 1.
template <int R0>
__device__ __forceinline__ void aes256_rounds_from(const AesSmem& S, const AesRK& rk, uint32_t& s0,
                                                   uint32_t& s1, uint32_t& s2, uint32_t& s3) {
#pragma unroll
    for (int r = R0; r < 14; r++) aes256_round(S, rk, r, s0, s1, s2, s3);
    // last round: S-box bytes read out of the T tables (T2 byte0, T3 byte1,
    // T0 byte2 and T1 byte3 all hold S[x])
    const uint32_t n0 = (S.lk<2, 0>(s0) & 0xffu) | (S.lk<3, 1>(s1) & 0xff00u) |
                        (S.lk<0, 2>(s2) & 0xff0000u) | (S.lk<1, 3>(s3) & 0xff000000u);
    const uint32_t n1 = (S.lk<2, 0>(s1) & 0xffu) | (S.lk<3, 1>(s2) & 0xff00u) |
                        (S.lk<0, 2>(s3) & 0xff0000u) | (S.lk<1, 3>(s0) & 0xff000000u);
    const uint32_t n2 = (S.lk<2, 0>(s2) & 0xffu) | (S.lk<3, 1>(s3) & 0xff00u) |
                        (S.lk<0, 2>(s0) & 0xff0000u) | (S.lk<1, 3>(s1) & 0xff000000u);
    const uint32_t n3 = (S.lk<2, 0>(s3) & 0xffu) | (S.lk<3, 1>(s0) & 0xff00u) |
                        (S.lk<0, 2>(s1) & 0xff0000u) | (S.lk<1, 3>(s2) & 0xff000000u);
    s0 = n0 ^ rk.k[56];
    s1 = n1 ^ rk.k[57];
    s2 = n2 ^ rk.k[58];
    s3 = n3 ^ rk.k[59];
}

// Encrypt one block (4 little-endian column words) in place.
__device__ __forceinline__ void aes256_encrypt(const AesSmem& S, const AesRK& rk, uint32_t& s0,
                                               uint32_t& s1, uint32_t& s2, uint32_t& s3) {
    s0 ^= rk.k[0];
    s1 ^= rk.k[1];
    s2 ^= rk.k[2];
    s3 ^= rk.k[3];
    aes256_rounds_from<1>(S, rk, s0, s1, s2, s3);
}

// Keystream block `blk` of a draw that starts at nonce `nonce0` of the stream
// keyed by rk.
__device__ __forceinline__ uint4 keystream_block_n(const AesSmem& S, const AesRK& rk,
                                                   unsigned long long nonce0, unsigned long long blk) {
    const unsigned long long nonce = nonce0 + (blk >> 16);
    uint32_t s0 = (uint32_t)nonce, s1 = (uint32_t)(nonce >> 32), s2 = 0u;
    uint32_t s3 = __byte_perm((uint32_t)(blk & 0xffffu) + 2u, 0, 0x0123);
    aes256_encrypt(S, rk, s0, s1, s2, s3);
    return make_uint4(s0, s1, s2, s3);
}

// Keystream block `blk` (16-byte unit) of a draw that starts at nonce `nonce0`.
__device__ __forceinline__ uint4 keystream_block(const AesSmem& S, const StreamArg& st,
                                                 unsigned long long blk) {
    const unsigned long long nonce = st.nonce + (blk >> 16);
    uint32_t s0 = (uint32_t)nonce, s1 = (uint32_t)(nonce >> 32), s2 = 0u;
    uint32_t s3 = __byte_perm((uint32_t)(blk & 0xffffu) + 2u, 0, 0x0123);
    aes256_encrypt(S, st.rk, s0, s1, s2, s3);
    return make_uint4(s0, s1, s2, s3);
}

// The first two rounds of a chunk's blocks without their constant parts (counter
// mode caching: Bernstein and Schwabe, New AES software speed records, 2008). GCM's
// counter block is (nonce, 0, BE32(j + 2)): in round 1 counter byte 15 reaches
// column 0, byte 14 column 1 and byte 13 (1 for the chunk's last two blocks,
// else 0) column 2, so round 2 is the XOR of two table words a column and a
// constant of (key, nonce, byte 13). 10 lookups and two broadcast loads in
// place of 32 lookups: 0.91 of a block's shared-memory cycles.
struct __align__(16) CtrPre {
    uint32_t c0, c1, pad0, pad1;  // columns 0 and 1 of round 1 without bytes 15 and 14
    uint32_t k[4];                // round 2 without columns 0 and 1 of round 1
};

__device__ __forceinline__ CtrPre ctr_pre(const AesSmem& S, const AesRK& rk, unsigned long long nonce, uint32_t byte13) {
    const uint32_t w0 = (uint32_t)nonce ^ rk.k[0], w1 = (uint32_t)(nonce >> 32) ^ rk.k[1], w2 = rk.k[2];
    const uint32_t w3 = (byte13 << 8) ^ rk.k[3];
    const uint32_t n2 = S.lk<0, 0>(w2) ^ S.lk<1, 1>(w3) ^ S.lk<2, 2>(w0) ^ S.lk<3, 3>(w1) ^ rk.k[6];
    const uint32_t n3 = S.lk<0, 0>(w3) ^ S.lk<1, 1>(w0) ^ S.lk<2, 2>(w1) ^ S.lk<3, 3>(w2) ^ rk.k[7];
    CtrPre r;
    r.c0 = S.lk<0, 0>(w0) ^ S.lk<1, 1>(w1) ^ S.lk<2, 2>(w2) ^ rk.k[4];
    r.c1 = S.lk<0, 0>(w1) ^ S.lk<1, 1>(w2) ^ S.lk<3, 3>(w0) ^ rk.k[5];
    r.pad0 = r.pad1 = 0;
    r.k[0] = S.lk<2, 2>(n2) ^ S.lk<3, 3>(n3) ^ rk.k[8];
    r.k[1] = S.lk<1, 1>(n2) ^ S.lk<2, 2>(n3) ^ rk.k[9];
    r.k[2] = S.lk<0, 0>(n2) ^ S.lk<1, 1>(n3) ^ rk.k[10];
    r.k[3] = S.lk<0, 0>(n3) ^ S.lk<3, 3>(n2) ^ rk.k[11];
    return r;
}

// Block `blk` of a draw that starts at nonce `nonce0`. With the constants of
// its chunk in pre[0] (byte 13 = 0) and pre[1] (byte 13 = 1), or without
// (null); both share the code of rounds 3 to 14: how much code a loop holds
// decides its speed (the instruction cache), and a short call's latency.
__device__ __forceinline__ uint4 keystream_block_pre(const AesSmem& S, const AesRK& rk, const CtrPre* pre,
                                                     unsigned long long nonce0, unsigned long long blk) {
    const uint32_t ctr = ((uint32_t)blk & 0xffffu) + 2;
    uint32_t s0, s1, s2, s3;
    const uint32_t w3 = __byte_perm(ctr, 0, 0x0123) ^ rk.k[3];
    if (pre) {
        const CtrPre* q = pre + (ctr >> 16);
        const uint2 c = *reinterpret_cast<const uint2*>(q);
        const uint4 k = *reinterpret_cast<const uint4*>(q->k);
        const uint32_t n0 = c.x ^ S.lk<3, 3>(w3), n1 = c.y ^ S.lk<2, 2>(w3);
        s0 = k.x ^ S.lk<0, 0>(n0) ^ S.lk<1, 1>(n1);
        s1 = k.y ^ S.lk<0, 0>(n1) ^ S.lk<3, 3>(n0);
        s2 = k.z ^ S.lk<2, 2>(n0) ^ S.lk<3, 3>(n1);
        s3 = k.w ^ S.lk<1, 1>(n0) ^ S.lk<2, 2>(n1);
    } else {
        const unsigned long long nonce = nonce0 + (blk >> 16);
        s0 = (uint32_t)nonce ^ rk.k[0];
        s1 = (uint32_t)(nonce >> 32) ^ rk.k[1];
        s2 = rk.k[2];
        s3 = w3;
#pragma unroll
        for (int r = 1; r < 3; r++) aes256_round(S, rk, r, s0, s1, s2, s3);
    }
    aes256_rounds_from<3>(S, rk, s0, s1, s2, s3);
    return make_uint4(s0, s1, s2, s3);
}

}  // namespace orqcu
