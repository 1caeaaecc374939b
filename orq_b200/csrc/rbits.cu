// rbits.cu — the bit loop of radix_sort (include/core/operators/radixsort.h:
// 116-203) as one cooperative kernel. Per bit: bit_arithmetic_right_shift and
// b2a_bit of the bit (f1), prefix_sum of s = [1 - f1, f1] with s[0] -= 1,
// t = s0 + f1 * (s1 - s0), oblivious_apply_elementwise_perm(rows, t).
//
// A bit is five phases with a grid barrier after each: b2a of the bit, the
// destination multiply (its scan needs every CTA's sum of the flags), and the
// three groups' gather + reshare, the last of which opens the destinations and
// scatters the rows. The AES tables are staged once; a phase's keystream does
// not depend on data and is computed before its barrier is waited for. Bound:
// launches below ~2^15 rows (eight of 5 to 10 us a bit before, now five
// barriers), the T-table lookups and the row gathers above. All bits of 40,
// int64 keys, eight launches a bit and now: 1000 rows 3.3 (host-bound) and
// 0.70 ms, 100003 rows 8.0 and 2.0, 2^20 rows 26.4 and 17.8, 2^22 rows 107.5
// and 71.9. A pass of 1024 rows with one keystream buffer: two buffers (one
// barrier a pass) or 512 rows leave the gathers less L1 and took 5-9 % longer.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "launch.cuh"

namespace orqcu {

namespace {

constexpr int kThreads = 512;
constexpr uint32_t kPass = 1024;  // elements of a CTA's pass
constexpr int kMaxBits = 64;
// keystream of a pass: 9 int32 calls (b2a), or two of the row and two of the
// destination shares (at most 40 bytes an element)
constexpr size_t kSmem = kAesSmemBytes + (size_t)kPass * 40;

// A row in the kernel is one 64-byte record: its three key shares (PW bytes
// each), then the three int32 shares of its destination. A gather of a row is
// two whole sectors (six half-used ones with the shares in arrays of their
// own), loaded by four lanes, 16 bytes each.
constexpr uint32_t kRec = 64;
constexpr uint32_t kPieces = kPass * 4 / kThreads;  // 16-byte pieces a thread moves per pass

struct BitsArgs {
    void* P[3];       // padded rows, in and out
    uint8_t* rec[2];  // [n] records
    uint32_t* f1[3];  // the bit's A-shares
    uint32_t* part;   // [2][grid][3] sums of f1 per CTA, by parity of the bit
    uint32_t* bar;    // arrivals, counted from 0
    int* err;
    const int32_t* inv[3 * kMaxBits];  // [bit][group] inverse local permutations
    AesRK rk[6];                       // PAIR0..2, G01, G02, G12
    unsigned long long nonce[6];
    unsigned long long ch4, chx;       // nonces of an n-element int32 / row call
    uint32_t n, chunk, bits, invert_last;
};

template <int PW>
__global__ void __launch_bounds__(kThreads, 1) k_radix_bits(BitsArgs a) {
    using R = Ring<4>;
    constexpr uint32_t kRowsPerBlk = 16 / PW;
    extern __shared__ __align__(16) uint32_t sm[];
    __shared__ uint32_t red[3][kThreads / 32], sbase[3], stot[3];
    __shared__ int s_dead;
    aes_stage_tables(sm);
    const AesSmem S(sm);
    uint4* ks = reinterpret_cast<uint4*>(sm + kAesSmemBytes / 4);
    const uint32_t* kw = reinterpret_cast<const uint32_t*>(ks);
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const uint32_t c0 = blockIdx.x * a.chunk, c1 = min(a.n, c0 + a.chunk);
    const uint32_t G = gridDim.x;
    const unsigned long long nb4 = 4ull * a.n;
    uint32_t target = 0;  // arrivals that open the next phase
    if (tid == 0) s_dead = 0;
    // the phase before is complete everywhere (thread 0 waits for all)
    const auto wait = [&]() {
        if (tid != 0 || !target) return;
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
    };
    const uint32_t pc = tid & 3;  // this thread's piece of every record it moves
    int cur = 0;                  // rows of the bit are in a.rec[cur]
    for (uint32_t e = c0 + tid; e < c1; e += kThreads) {
        uint8_t* r = a.rec[0] + (size_t)e * kRec;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            if constexpr (PW == 16)
                reinterpret_cast<uint4*>(r)[j] = __ldcg(reinterpret_cast<const uint4*>(a.P[j]) + e);
            else
                reinterpret_cast<uint2*>(r)[j] = __ldcg(reinterpret_cast<const uint2*>(a.P[j]) + e);
        }
    }
    __syncthreads();
    for (uint32_t bit = 0; bit < a.bits; bit++) {
        const uint32_t wsel = (32 + bit) >> 5, bsel = bit & 31;
        const uint32_t invert = (a.invert_last && bit + 1 == a.bits) ? 1u : 0u;
        uint32_t* part = a.part + (size_t)(bit & 1) * 3 * G;
        uint32_t run[3] = {0, 0, 0};  // phase 0: this CTA's sums; phase 1: prefixes
        for (int ph = 0; ph < 5; ph++) {
            for (uint32_t e0 = c0; e0 < c1; e0 += kPass) {
                const uint32_t ne = min(kPass, c1 - e0);  // elements of the pass
                const uint32_t nu = (ne + 3) / 4;         // int32 blocks
                // ---- rows of the pass: indices now; the gathers as early as the
                // barrier allows, so that they arrive during the keystream
                const uint8_t* src = a.rec[ph == 3 ? cur ^ 1 : cur];
                uint32_t id[kPieces];
                uint4 v[kPieces];
                const auto gather = [&]() {
#pragma unroll
                    for (uint32_t r = 0; r < kPieces; r++)
                        if (kThreads / 4 * r + tid / 4 < ne && (PW == 16 || pc != 3))
                            v[r] = __ldcg(reinterpret_cast<const uint4*>(src + (size_t)id[r] * kRec) + pc);
                };
                if (ph >= 2) {
                    const int32_t* idx = a.inv[3 * bit + ph - 2];
#pragma unroll
                    for (uint32_t r = 0; r < kPieces; r++) {
                        const uint32_t e = kThreads / 4 * r + tid / 4;
                        id[r] = e < ne ? (uint32_t)__ldg(idx + e0 + e) : 0u;
                    }
                    if (e0 != c0) gather();
                }
                // ---- keystream of the pass
                const uint32_t nk = ph < 2 ? 0u : (ne + kRowsPerBlk - 1) / kRowsPerBlk;
                const uint32_t total = ph == 0 ? 9 * nu : (ph == 1 ? 3 * nu : 2 * nk + 2 * nu);
                for (uint32_t i = tid; i < total; i += kThreads) {
                    uint32_t s;
                    unsigned long long nonce, blk = e0 / 4;
                    if (ph < 2) {
                        const uint32_t f = i / nu;
                        s = f % 3;
                        nonce = a.nonce[s] + (4ull * bit + (ph == 0 ? f / 3 : 3u)) * a.ch4;
                        blk += i - f * nu;
                    } else {
                        s = 1 + ph;
                        nonce = a.nonce[s] + bit * (2 * a.chx + 2 * a.ch4);
                        if (i < 2 * nk) {
                            const uint32_t f = i >= nk;
                            nonce += f ? a.chx : 0ull;
                            blk = e0 / kRowsPerBlk + (i - f * nk);
                        } else {
                            const uint32_t j = i - 2 * nk, f = j >= nu;
                            nonce += 2 * a.chx + (f ? a.ch4 : 0ull);
                            blk += j - f * nu;
                        }
                    }
                    ks[i] = keystream_block_n(S, a.rk[s], nonce, blk);
                }
                if (e0 == c0) {
                    wait();
                    __syncthreads();
                    if (s_dead) return;  // uniform: written before the barrier above
                    if (ph >= 2) gather();
                } else {
                    __syncthreads();
                }
                if (ph == 0) {
                    uint32_t sum[3] = {0, 0, 0};
                    if (tid < nu) {
                        uint4 z[3][3];
#pragma unroll
                        for (int c = 0; c < 3; c++) {
                            const uint4 k0 = ks[(3 * c + 0) * nu + tid], k1 = ks[(3 * c + 1) * nu + tid],
                                        k2 = ks[(3 * c + 2) * nu + tid];
                            z[c][0] = R::sub(k2, k0);
                            z[c][1] = R::sub(k0, k1);
                            z[c][2] = R::sub(k1, k2);
                        }
                        uint32_t x[3][4];
#pragma unroll
                        for (int j = 0; j < 3; j++)
#pragma unroll
                            for (int e = 0; e < 4; e++) {
                                const uint32_t i = e0 + 4 * tid + e;
                                const uint32_t b =
                                    i < c1 ? __ldcg(reinterpret_cast<const uint32_t*>(src + (size_t)i * kRec + j * PW) + wsel)
                                           : 0u;
                                x[j][e] = ((b >> bsel) ^ invert) & 1u;
                            }
                        const uint4 abit = make_uint4(x[0][0] ^ x[1][0], x[0][1] ^ x[1][1], x[0][2] ^ x[1][2],
                                                      x[0][3] ^ x[1][3]);
                        const uint4 bbit = make_uint4(x[2][0], x[2][1], x[2][2], x[2][3]);
                        uint4 d[3];
                        d[0] = R::sub(R::add(z[0][0], abit), z[1][0]);
                        d[1] = R::sub(z[0][1], R::add(z[1][1], bbit));
                        d[2] = R::sub(z[0][2], z[1][2]);
                        const uint32_t left = c1 - (e0 + 4 * tid);
#pragma unroll
                        for (int p = 0; p < 3; p++) {
                            const int q = (p + 1) % 3;
                            uint4 v = R::add(z[2][p], R::mul(d[p], d[p]));
                            v = R::add(v, R::mul(d[p], d[q]));
                            v = R::add(v, R::mul(d[q], d[p]));
                            st16(a.f1[p], e0 / 4 + tid, nb4, v);
                            sum[p] = v.x + (left > 1 ? v.y : 0u) + (left > 2 ? v.z : 0u) + (left > 3 ? v.w : 0u);
                        }
                    }
#pragma unroll
                    for (int p = 0; p < 3; p++) run[p] += sum[p];
                } else if (ph == 1) {
                    if (e0 == c0) {
                        // the sums of the CTAs before this one, and of all
                        if (w < 3) {
                            uint32_t b = 0, t = 0;
                            for (uint32_t k = lane; k < G; k += 32) {
                                const uint32_t v = __ldcg(part + 3 * k + w);
                                t += v;
                                b += k < blockIdx.x ? v : 0u;
                            }
                            b = __reduce_add_sync(0xffffffffu, b);
                            t = __reduce_add_sync(0xffffffffu, t);
                            if (lane == 0) {
                                sbase[w] = b;
                                stot[w] = t;
                            }
                        }
                        __syncthreads();
#pragma unroll
                        for (int p = 0; p < 3; p++) run[p] = sbase[p];
                    }
                    uint4 x[3];
                    uint32_t inc[3], own[3];
#pragma unroll
                    for (int p = 0; p < 3; p++) {
                        x[p] = make_uint4(0, 0, 0, 0);
                        if (tid < nu) {
                            const uint32_t* f = a.f1[p] + e0 + 4 * tid;
                            const uint32_t left = c1 - (e0 + 4 * tid);
                            x[p].x = f[0];
                            if (left > 1) x[p].y = f[1];
                            if (left > 2) x[p].z = f[2];
                            if (left > 3) x[p].w = f[3];
                        }
                        own[p] = x[p].x + x[p].y + x[p].z + x[p].w;
                        inc[p] = own[p];
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const uint32_t y = __shfl_up_sync(0xffffffffu, inc[p], o);
                            if ((int)lane >= o) inc[p] += y;
                        }
                        if (lane == 31) red[p][w] = inc[p];
                    }
                    __syncthreads();
                    uint4 s0[3], y[3];
#pragma unroll
                    for (int p = 0; p < 3; p++) {
                        uint32_t pre = run[p] + inc[p] - own[p];
                        for (uint32_t k = 0; k < kThreads / 32; k++) {
                            const uint32_t v = red[p][k];
                            if (k < w) pre += v;
                            run[p] += v;
                        }
                        // F = inclusive prefix of f1; the scan of [1 - f1, f1] with
                        // s[0] -= 1 is i - F in the first half (the public i in
                        // share 0) and (n - 1, share 0) - total + F in the second
                        const uint4 F = make_uint4(pre + x[p].x, pre + x[p].x + x[p].y, pre + x[p].x + x[p].y + x[p].z,
                                                   pre + own[p]);
                        const uint32_t i = e0 + 4 * tid;
                        const uint4 pub = p == 0 ? make_uint4(i, i + 1, i + 2, i + 3) : make_uint4(0, 0, 0, 0);
                        const uint32_t half = (p == 0 ? a.n - 1 : 0u) - stot[p];
                        s0[p] = R::sub(pub, F);
                        y[p] = R::sub(R::add(make_uint4(half, half, half, half), F), s0[p]);
                    }
                    if (tid < nu) {
                        const uint4 k0 = ks[tid], k1 = ks[nu + tid], k2 = ks[2 * nu + tid];
                        const uint4 r[3] = {R::sub(k2, k0), R::sub(k0, k1), R::sub(k1, k2)};
#pragma unroll
                        for (int p = 0; p < 3; p++) {
                            const int q = (p + 1) % 3;
                            uint4 v = R::add(r[p], R::mul(x[p], y[p]));
                            v = R::add(v, R::mul(x[p], y[q]));
                            v = R::add(v, R::mul(x[q], y[p]));
                            v = R::add(s0[p], v);
                            const uint32_t t[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                            for (int e = 0; e < 4; e++)
                                if (e0 + 4 * tid + e < c1)
                                    reinterpret_cast<uint32_t*>(a.rec[cur] + (size_t)(e0 + 4 * tid + e) * kRec + 3 * PW)[p] = t[e];
                        }
                    }
                } else {
                    uint8_t* dst = a.rec[ph == 3 ? cur : cur ^ 1];
                    const uint32_t* q0 = kw + 4 * (2 * nk);  // destination shares' keystream
                    const uint32_t* q1 = q0 + 4 * nu;
#pragma unroll
                    for (uint32_t r = 0; r < kPieces; r++) {
                        const uint32_t e = kThreads / 4 * r + tid / 4;
                        const bool in = e < ne;
                        uint4 x = v[r];
                        uint32_t t = 0;  // this piece's part of the opened destination
                        if (in) {
                            if constexpr (PW == 16) {
                                if (pc == 3) {
                                    x.x += q0[e];
                                    x.y += q1[e];
                                    x.z -= q0[e] + q1[e];
                                    t = x.x + x.y + x.z;
                                } else {
                                    if (pc != 1) x = x ^ ks[e];
                                    if (pc != 0) x = x ^ ks[nk + e];
                                }
                            } else {
                                const uint2 r0 = reinterpret_cast<const uint2*>(ks)[e];
                                const uint2 r1 = reinterpret_cast<const uint2*>(ks + nk)[e];
                                if (pc == 0) {
                                    x = x ^ make_uint4(r0.x, r0.y, r1.x, r1.y);
                                } else if (pc == 1) {
                                    x.x ^= r0.x ^ r1.x;
                                    x.y ^= r0.y ^ r1.y;
                                    x.z += q0[e];
                                    x.w += q1[e];
                                    t = x.z + x.w;
                                } else {
                                    x.x -= q0[e] + q1[e];
                                    t = pc == 2 ? x.x : 0u;
                                }
                            }
                        }
                        uint32_t o = e0 + e;
                        if (ph == 4) {
                            // the opened destination, from the record's lanes
                            if constexpr (PW == 16) {
                                o = __shfl_sync(0xffffffffu, t, lane | 3);
                            } else {
                                o = __shfl_sync(0xffffffffu, t, (lane & ~3u) | 1) + __shfl_sync(0xffffffffu, t, (lane & ~3u) | 2);
                            }
                            if (in && o >= a.n) {  // corrupted shares: flag, skip the store
                                atomicOr(a.err, 8);
                                continue;
                            }
                        }
                        if (in && (PW == 16 || pc != 3)) reinterpret_cast<uint4*>(dst + (size_t)o * kRec)[pc] = x;
                    }
                }
                __syncthreads();  // the next pass rewrites the keystream
            }
            if (ph == 0) {
#pragma unroll
                for (int p = 0; p < 3; p++) {
                    const uint32_t s = __reduce_add_sync(0xffffffffu, run[p]);
                    if (lane == 0) red[p][w] = s;
                }
                __syncthreads();
                if (tid < 3) {
                    uint32_t s = 0;
                    for (int k = 0; k < kThreads / 32; k++) s += red[tid][k];
                    part[3 * blockIdx.x + tid] = s;
                }
            }
            target += G;
            __syncthreads();
            if (tid == 0) {
                __threadfence();
                asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
            }
        }
        cur ^= 1;
    }
    wait();
    __syncthreads();
    if (s_dead) return;
    for (uint32_t e = c0 + tid; e < c1; e += kThreads) {
        const uint8_t* r = a.rec[cur] + (size_t)e * kRec;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            if constexpr (PW == 16)
                reinterpret_cast<uint4*>(a.P[j])[e] = __ldcg(reinterpret_cast<const uint4*>(r) + j);
            else
                reinterpret_cast<uint2*>(a.P[j])[e] = __ldcg(reinterpret_cast<const uint2*>(r) + j);
        }
    }
}

}  // namespace

// Runs `bits` bit passes on the padded rows P with the next `bits` reserved
// permutations (the caller has reserved them).
void op_radix_bits(Ctx& c, int PW, size_t n, Sh3 P, int bits, bool invert_last) {
    if (bits > kMaxBits || (PW != 8 && PW != 16)) throw std::invalid_argument("bits out of range");
    if (!n) {  // the queue moves on and no stream does
        for (int b = 0; b < bits; b++) {
            ShardedPerm sp = next_perm(c, n);
            c.free_perm(sp);
        }
        return;
    }
    const uint32_t sms = (uint32_t)std::max(1, c.num_sms);
    // chunks of whole 64-element groups keep every stream's blocks inside one CTA
    const uint32_t chunk = (uint32_t)(ceil_div(ceil_div(n, sms), 64) * 64);
    const uint32_t grid = (uint32_t)ceil_div(n, chunk);
    const size_t n4 = ceil_div(n, 4) * 4;  // 16-byte aligned share arrays
    Scratch recs(c, 2 * n * kRec), f1b(c, 3 * n4 * 4), part(c, (size_t)6 * grid * 4);
    BitsArgs a;
    for (int j = 0; j < 3; j++) {
        a.P[j] = P.p[j];
        a.f1[j] = f1b.as<uint32_t>() + j * n4;
        a.rk[j] = c.rk[PAIR0 + j];
        a.nonce[j] = c.nonce[PAIR0 + j];
        a.rk[3 + j] = c.rk[G01 + j];
        a.nonce[3 + j] = c.nonce[G01 + j];
    }
    a.rec[0] = recs.as<uint8_t>();
    a.rec[1] = a.rec[0] + n * kRec;
    a.part = part.as<uint32_t>();
    a.bar = c.grid_bar();
    a.err = c.d_err;
    a.ch4 = chunks_of((unsigned long long)n * 4);
    a.chx = chunks_of((unsigned long long)n * PW);
    a.n = (uint32_t)n;
    a.chunk = chunk;
    a.bits = (uint32_t)bits;
    a.invert_last = invert_last;
    std::vector<ShardedPerm> used;
    for (int b = 0; b < bits; b++) {
        used.push_back(next_perm(c, n));
        for (int g = 0; g < 3; g++) a.inv[3 * b + g] = used.back().inv[g];
    }
    ORQ_CUDA_CHECK(cudaMemsetAsync(a.bar, 0, 4, c.stream));
    {
        const double el = (double)n * bits;
        ProfScope ps(c, "radix_bits", el * (24.0 + 24.0 + 3 * (4.0 + 6.0 * PW + 24.0)),
                     el * (9.0 / 4 + 3.0 / 4 + 6.0 * (PW / 16.0 + 0.25)));
        void* args[] = {&a};
        const auto kern = PW == 16 ? &k_radix_bits<16> : &k_radix_bits<8>;
        ORQ_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
        ORQ_CUDA_CHECK(cudaLaunchCooperativeKernel((const void*)kern, dim3(grid), dim3(kThreads), args, kSmem, c.stream));
    }
    c.kernels_launched++;
    for (auto& sp : used) c.free_perm(sp);
    for (int q = 0; q < 3; q++) {
        c.nonce[PAIR0 + q] += 4ull * bits * a.ch4;
        c.nonce[G01 + q] += (unsigned long long)bits * (2 * a.chx + 2 * a.ch4);
    }
}

}  // namespace orqcu
