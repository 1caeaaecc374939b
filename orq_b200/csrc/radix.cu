// radix.cu — ORQ's shuffle-based oblivious radix sort on the loopback runtime.
//
// Restates orq::operators::radix_sort (include/core/operators/radixsort.h:
// 116-229) with pad_input / remove_padding (operators/sorting.h:405-495) and
// ElementwisePermutation::b2a / invert (containers/permutation.h:205-258),
// calling the same protocol steps in the same order so every PRG stream is
// consumed exactly as the reference consumes it. The bit loop is rbits.cu.
#include <algorithm>
#include <functional>
#include <numeric>
#include <vector>

#include "launch.cuh"

namespace orqcu {

namespace {

// pad_input (sorting.h:431-462): (v << 32) | index, index public-shared into
// S0 only (P0 and P2 hold it); v is sign-extended to the padded width.
// Descending (reverse_order): the index is -1-i and the padded vector is
// reversed, so row i lands at position n-1-i.
template <int KW, int PW>
__global__ void k_pad(CSh3 key, Sh3 P, unsigned long long n, int desc) {
    for (unsigned long long i0 = gtid(); i0 < n; i0 += gstride()) {
        const unsigned long long i = desc ? n - 1 - i0 : i0;  // destination
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const uint32_t idx = j == 0 ? (desc ? (uint32_t)(-1ll - (long long)i0) : (uint32_t)i0) : 0u;
            if constexpr (KW == 8) {
                const long long v = reinterpret_cast<const long long*>(key.p[j])[i0];
                const unsigned long long lo = ((unsigned long long)v << 32) | idx;
                const unsigned long long hi = (unsigned long long)(v >> 32);  // sign fill
                reinterpret_cast<uint4*>(P.p[j])[i] = mk4(lo, hi);
            } else {
                const int v = reinterpret_cast<const int*>(key.p[j])[i0];
                const unsigned long long p = ((unsigned long long)(long long)v << 32) | idx;
                reinterpret_cast<unsigned long long*>(P.p[j])[i] = p;
            }
        }
    }
}

// remove_padding (sorting.h:475-495): low 32 bits -> B-shared permutation,
// arithmetic shift by 32 -> the key.
// Descending: the padded vector is reversed back first (row i reads n-1-i).
template <int KW, int PW>
__global__ void k_unpad(CSh3 P, Sh3 key, Sh3 perm, unsigned long long n, int desc) {
    for (unsigned long long i = gtid(); i < n; i += gstride()) {
        const unsigned long long src = desc ? n - 1 - i : i;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            if constexpr (PW == 16) {
                const uint4 v = reinterpret_cast<const uint4*>(P.p[j])[src];
                reinterpret_cast<uint32_t*>(perm.p[j])[i] = v.x;
                const unsigned long long k = (unsigned long long)v.y | ((unsigned long long)v.z << 32);
                reinterpret_cast<unsigned long long*>(key.p[j])[i] = k;
            } else {
                const unsigned long long v = reinterpret_cast<const unsigned long long*>(P.p[j])[src];
                reinterpret_cast<uint32_t*>(perm.p[j])[i] = (uint32_t)v;
                reinterpret_cast<uint32_t*>(key.p[j])[i] = (uint32_t)(v >> 32);
            }
        }
    }
}

__global__ void k_iota(int32_t* out, unsigned long long n) {
    for (unsigned long long i = gtid(); i < n; i += gstride()) out[i] = (int32_t)i;
}

// public_share of the constant -1 (S0 = -1, S1 = S2 = 0)
__global__ void k_minus_one(Sh3 m, unsigned long long n) {
    for (unsigned long long i = gtid(); i < n; i += gstride()) {
        reinterpret_cast<int32_t*>(m.p[0])[i] = -1;
        reinterpret_cast<int32_t*>(m.p[1])[i] = 0;
        reinterpret_cast<int32_t*>(m.p[2])[i] = 0;
    }
}

}  // namespace

// The frame both sort protocols share (radix_sort, radixsort.h:205-229, and
// quicksort, quicksort.h:214-246): pad_input, the protocol's body on the
// padded rows, remove_padding (permutation b2a, negate for descending order)
// and invert. `reserve` is the number of permutations the body and the frame
// take from the PermutationManager queue, reserved up front.
void sort_padded(Ctx& c, int kw, size_t n, Sh3 key, bool desc, Sh3 perm_out, size_t reserve,
                 const std::function<void(Sh3 P, int PW)>& body) {
    if (kw != 4 && kw != 8) throw std::invalid_argument("sort keys must be int32 or int64");
    if (n >= (1ull << 31)) throw std::invalid_argument("sorts support n < 2^31");
    const int PW = kw == 8 ? 16 : 8;
    reserve_perms(c, n, reserve);

    Scratch Pbuf(c, 3 * std::max<size_t>(n, 1) * PW);
    Sh3 P;
    for (int j = 0; j < 3; j++) P.p[j] = Pbuf.as<uint8_t>() + j * n * (size_t)PW;
    const unsigned pg = plain_grid(c, n);
    if (n) {
        CSh3 k{{key.p[0], key.p[1], key.p[2]}};
        if (kw == 8) k_pad<8, 16><<<pg, 256, 0, c.stream>>>(k, P, n, desc);
        else k_pad<4, 8><<<pg, 256, 0, c.stream>>>(k, P, n, desc);
        ORQ_CUDA_CHECK(cudaGetLastError());
        c.kernels_launched++;
    }
    body(P, PW);
    const size_t n1 = std::max<size_t>(n, 1);

    // remove_padding: permutation = low 32 bits (B-shared), key = padded >> 32
    Scratch pm(c, 3 * n1 * 4);
    Sh3 PM;
    for (int j = 0; j < 3; j++) PM.p[j] = pm.as<uint8_t>() + j * n1 * 4;
    if (n) {
        CSh3 Pc{{P.p[0], P.p[1], P.p[2]}};
        if (kw == 8) k_unpad<8, 16><<<pg, 256, 0, c.stream>>>(Pc, key, PM, n, desc);
        else k_unpad<4, 8><<<pg, 256, 0, c.stream>>>(Pc, key, PM, n, desc);
        ORQ_CUDA_CHECK(cudaGetLastError());
        c.kernels_launched++;
    }

    // ElementwisePermutation::b2a (permutation.h:222-258): shuffle a copy with
    // pi, open it, public-share it arithmetically, un-apply pi.
    {
        ShardedPerm sp = next_perm(c, n);
        Scratch pcb(c, 3 * n1 * 4), sig(c, n1 * 4);
        Sh3 PC;
        for (int j = 0; j < 3; j++) {
            PC.p[j] = pcb.as<uint8_t>() + j * n1 * 4;
            if (n)
                ORQ_CUDA_CHECK(cudaMemcpyAsync(PC.p[j], PM.p[j], n * 4, cudaMemcpyDeviceToDevice, c.stream));
        }
        op_apply_sharded(c, false, 4, n, PC, sp, false);
        op_open(c, false, 4, n, CSh3{{PC.p[0], PC.p[1], PC.p[2]}}, sig.p);
        op_public_share(c, 4, n, sig.p, PM);
        op_apply_sharded(c, true, 4, n, PM, sp, true);
        c.free_perm(sp);
    }
    // negate (permutation.h:268-280) for descending sorts: v *= -1 (a
    // multiply_a with the public -1), v += -1
    if (desc) {
        Scratch mb(c, 3 * n1 * 4);
        Sh3 M1;
        for (int j = 0; j < 3; j++) M1.p[j] = mb.as<uint8_t>() + j * n1 * 4;
        if (n) {
            k_minus_one<<<pg, 256, 0, c.stream>>>(M1, n);
            ORQ_CUDA_CHECK(cudaGetLastError());
            c.kernels_launched++;
        }
        const CSh3 m1c{{M1.p[0], M1.p[1], M1.p[2]}};
        op_mult(c, true, 4, n, CSh3{{PM.p[0], PM.p[1], PM.p[2]}}, m1c, PM);
        op_local(c, 1, 4, n, CSh3{{PM.p[0], PM.p[1], PM.p[2]}}, m1c, PM);
    }
    // invert (permutation.h:205-213): apply the permutation to a public identity
    {
        Scratch inv(c, 3 * n1 * 4);
        Sh3 I;
        for (int j = 0; j < 3; j++) I.p[j] = inv.as<uint8_t>() + j * n1 * 4;
        if (n) {
            k_iota<<<pg, 256, 0, c.stream>>>((int32_t*)I.p[0], n);
            ORQ_CUDA_CHECK(cudaGetLastError());
            c.kernels_launched++;
        }
        op_public_share(c, 4, n, I.p[0], I);
        op_apply_elementwise(c, true, 4, n, I, CSh3{{PM.p[0], PM.p[1], PM.p[2]}});
        for (int j = 0; j < 3; j++)
            if (n)
                ORQ_CUDA_CHECK(cudaMemcpyAsync(perm_out.p[j], I.p[j], n * 4, cudaMemcpyDeviceToDevice, c.stream));
    }
}

void op_radix_sort(Ctx& c, int kw, size_t n, Sh3 key, int bits, bool desc, Sh3 perm_out) {
    if (kw != 4 && kw != 8) throw std::invalid_argument("radix sort keys must be int32 or int64");
    if (bits < 1 || bits > kw * 8) throw std::invalid_argument("bits out of range");
    const bool full_width = (kw * 8 == bits);
    // radix_sort_body: 1 permutation for remove_padding + (bits + 1) pairs
    sort_padded(c, kw, n, key, desc, perm_out, (size_t)bits + 2,
                [&](Sh3 P, int PW) { op_radix_bits(c, PW, n, P, bits, full_width); });
}

// ---------------------------------------------------------------------------
// Batched radix sorts: `count` items in list order, the shares of `count`
// plain calls. Items run back to back on the runtime's stream; the host waits
// for their permutations, and once at the end. Overlapping item k's bit
// passes with item k+1's permutations is allowed by the PRG order (they only
// need nonces the host knows once item k's are generated). With the one-CTA
// scanner of an earlier chain it made the ragged batch slower, on a second
// stream with or without a static SM split (both halves want every SM for AES);
// it has not been measured with the present generator.
void op_radix_sort_batch(Ctx& c, int kw, int count, const size_t* n, void* const* keys, const int* bits,
                         const int* desc, void* const* perms_out) {
    if (count <= 0) return;
    for (int k = 0; k < count; k++) {
        if (kw != 4 && kw != 8) throw std::invalid_argument("radix sort keys must be int32 or int64");
        if (bits[k] < 1 || bits[k] > kw * 8) throw std::invalid_argument("bits out of range");
        if (n[k] >= (1ull << 31)) throw std::invalid_argument("sorts support n < 2^31");
    }
    for (int k = 0; k < count; k++) {
        Sh3 key{{keys[3 * k], keys[3 * k + 1], keys[3 * k + 2]}};
        Sh3 po{{perms_out[3 * k], perms_out[3 * k + 1], perms_out[3 * k + 2]}};
        op_radix_sort(c, kw, n[k], key, bits[k], desc[k] != 0, po);
    }
    c.check_device_error();
}

}  // namespace orqcu
