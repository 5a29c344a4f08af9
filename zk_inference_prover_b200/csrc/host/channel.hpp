// Host-side Fiat-Shamir channel of the prover: Blake2s-256 (RFC 7693) with every digest word
// reduced mod 2^31-1, as the reference's Blake2sM31Channel
// (nitroo/crates/stwo/src/core/channel/blake2s.rs:20-141, core/vcs/blake2_hash.rs:73-118,
// core/vcs/blake2_merkle.rs:53-58). Hashes are held as 8 little-endian words.
#pragma once
#include <array>
#include <cstdint>
#include <cstring>
#include <vector>
#if defined(__x86_64__)
#include <immintrin.h>
#endif

#include "../m31.cuh"

namespace b200 {

using HashWords = std::array<uint32_t, 8>;

class Blake2sState {
  public:
    Blake2sState() {
        for (int i = 0; i < 8; i++) h_[i] = IV[i];
        h_[0] ^= 0x01010020u;
    }
    void update(const uint8_t* p, size_t n) {
        while (n) {
            if (fill_ == 64) { t_ += 64; compress(false); fill_ = 0; }
            size_t k = n < 64 - fill_ ? n : 64 - fill_;
            memcpy(buf_ + fill_, p, k);
            fill_ += k; p += k; n -= k;
        }
    }
    void update_words(const uint32_t* w, size_t n) {
#if defined(__BYTE_ORDER__) && __BYTE_ORDER__ == __ORDER_LITTLE_ENDIAN__
        update(reinterpret_cast<const uint8_t*>(w), 4 * n);  // the words' memory is their little-endian serialisation
#else
        for (size_t i = 0; i < n; i++) {
            uint8_t b[4] = {(uint8_t)w[i], (uint8_t)(w[i] >> 8), (uint8_t)(w[i] >> 16), (uint8_t)(w[i] >> 24)};
            update(b, 4);
        }
#endif
    }
    // Digest with every word taken mod 2^31-1 (the M31 variant of the hasher).
    HashWords finalize_m31() {
        t_ += fill_;
        memset(buf_ + fill_, 0, 64 - fill_);
        compress(true);
        HashWords out;
        for (int i = 0; i < 8; i++) {
            uint32_t w = h_[i], s = (w & zk::P) + (w >> 31);
            out[i] = s >= zk::P ? s - zk::P : s;
        }
        return out;
    }
  private:
    void compress(bool last) {
        uint32_t m[16];
#if defined(__BYTE_ORDER__) && __BYTE_ORDER__ == __ORDER_LITTLE_ENDIAN__
        memcpy(m, buf_, 64);
#else
        for (int i = 0; i < 16; i++)
            m[i] = (uint32_t)buf_[4 * i] | ((uint32_t)buf_[4 * i + 1] << 8) | ((uint32_t)buf_[4 * i + 2] << 16) | ((uint32_t)buf_[4 * i + 3] << 24);
#endif
        compress_scalar(m, last);
    }
  public:
    static constexpr uint32_t IV[8] = {0x6A09E667u, 0xBB67AE85u, 0x3C6EF372u, 0xA54FF53Au, 0x510E527Fu, 0x9B05688Cu, 0x1F83D9ABu, 0x5BE0CD19u};
    static constexpr uint8_t SIGMA[10][16] = {
        {0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15}, {14, 10, 4, 8, 9, 15, 13, 6, 1, 12, 0, 2, 11, 7, 5, 3},
        {11, 8, 12, 0, 5, 2, 15, 13, 10, 14, 3, 6, 7, 1, 9, 4}, {7, 9, 3, 1, 13, 12, 11, 14, 2, 6, 5, 10, 4, 0, 15, 8},
        {9, 0, 5, 7, 2, 4, 10, 15, 14, 1, 11, 12, 6, 8, 3, 13}, {2, 12, 6, 10, 0, 11, 8, 3, 4, 13, 7, 5, 15, 14, 1, 9},
        {12, 5, 1, 15, 14, 13, 4, 10, 0, 7, 6, 3, 9, 2, 8, 11}, {13, 11, 7, 14, 12, 1, 3, 9, 5, 0, 15, 4, 8, 6, 2, 10},
        {6, 15, 14, 9, 11, 3, 0, 8, 12, 2, 13, 7, 1, 4, 10, 5}, {10, 2, 8, 4, 7, 6, 1, 5, 15, 11, 9, 14, 3, 12, 13, 0}};
  private:
    static uint32_t rotr(uint32_t x, int k) { return (x >> k) | (x << (32 - k)); }
    template <int R>
    __attribute__((always_inline)) static inline void round_scalar(uint32_t* v, const uint32_t* m) {
        auto g = [&](int a, int b, int c, int d, uint32_t x, uint32_t y) __attribute__((always_inline)) {
            v[a] += v[b] + x; v[d] = rotr(v[d] ^ v[a], 16);
            v[c] += v[d];     v[b] = rotr(v[b] ^ v[c], 12);
            v[a] += v[b] + y; v[d] = rotr(v[d] ^ v[a], 8);
            v[c] += v[d];     v[b] = rotr(v[b] ^ v[c], 7);
        };
        constexpr const uint8_t* s = SIGMA[R];
        g(0, 4, 8, 12, m[s[0]], m[s[1]]);   g(1, 5, 9, 13, m[s[2]], m[s[3]]);
        g(2, 6, 10, 14, m[s[4]], m[s[5]]);  g(3, 7, 11, 15, m[s[6]], m[s[7]]);
        g(0, 5, 10, 15, m[s[8]], m[s[9]]);  g(1, 6, 11, 12, m[s[10]], m[s[11]]);
        g(2, 7, 8, 13, m[s[12]], m[s[13]]); g(3, 4, 9, 14, m[s[14]], m[s[15]]);
    }
    void compress_scalar(const uint32_t* m, bool last) {
        uint32_t v[16];
        for (int i = 0; i < 8; i++) { v[i] = h_[i]; v[8 + i] = IV[i]; }
        v[12] ^= (uint32_t)t_;
        v[13] ^= (uint32_t)(t_ >> 32);
        if (last) v[14] = ~v[14];
        round_scalar<0>(v, m); round_scalar<1>(v, m); round_scalar<2>(v, m); round_scalar<3>(v, m); round_scalar<4>(v, m);
        round_scalar<5>(v, m); round_scalar<6>(v, m); round_scalar<7>(v, m); round_scalar<8>(v, m); round_scalar<9>(v, m);
        for (int i = 0; i < 8; i++) h_[i] ^= v[i] ^ v[8 + i];
    }
    uint32_t h_[8];
    uint8_t buf_[64];
    size_t fill_ = 0;
    uint64_t t_ = 0;
};

// H(head || words || zero bytes up to `bytes`), reduced. What the channel hashes is a chain (every message starts with the digest before
// it), so the latency of a message bounds the host's share of a batched GKR proof (three blocks a layer and instance) and of an opening
// of tens of thousands of columns. A vector register per row of the state makes each half round thirteen dependent instructions (the
// processors a B200 comes with have the rotate and the table permute), and blocks go from where they lie straight into registers:
// through a buffer every block waited twice for its own stores. 96 bytes: 236 ns, 285 ns through the buffer, 380-520 ns with rolled
// scalar rounds; elsewhere the rounds are unrolled on scalars.
#if defined(__x86_64__)
#define B200_ROWS __attribute__((target("avx512f,avx512vl,avx2")))
struct Blake2sRows {
    // The message words of a round in the order the rows take them: x and y of the four column steps, then of the four diagonal
    // steps as they lie when rows a, c and d have been turned and row b has not.
    struct alignas(64) Order {
        uint32_t w[10][16];
        Order() {
            for (int r = 0; r < 10; r++)
                for (int q = 0; q < 4; q++) {
                    const int diag = (q + 3) & 3;
                    const uint8_t* s = Blake2sState::SIGMA[r];
                    w[r][q] = s[2 * q];
                    w[r][4 + q] = s[2 * q + 1];
                    w[r][8 + q] = s[8 + 2 * diag];
                    w[r][12 + q] = s[9 + 2 * diag];
                }
        }
    };
    static bool here() {
        static const bool yes = __builtin_cpu_supports("avx512f") && __builtin_cpu_supports("avx512vl") && __builtin_cpu_supports("avx2");
        return yes;
    }
    B200_ROWS static inline void half_round(__m128i& a, __m128i& b, __m128i& c, __m128i& d, __m128i x, __m128i y) {
        a = _mm_add_epi32(_mm_add_epi32(a, x), b); d = _mm_ror_epi32(_mm_xor_si128(d, a), 16);
        c = _mm_add_epi32(c, d);                   b = _mm_ror_epi32(_mm_xor_si128(b, c), 12);
        a = _mm_add_epi32(_mm_add_epi32(a, y), b); d = _mm_ror_epi32(_mm_xor_si128(d, a), 8);
        c = _mm_add_epi32(c, d);                   b = _mm_ror_epi32(_mm_xor_si128(b, c), 7);
    }
    B200_ROWS static HashWords hash(const uint32_t* head, const uint32_t* words, size_t n, uint64_t bytes) {
        static const Order order;
        const __m128i iv0 = _mm_loadu_si128((const __m128i*)Blake2sState::IV), iv1 = _mm_loadu_si128((const __m128i*)(Blake2sState::IV + 4));
        __m128i h0 = _mm_xor_si128(iv0, _mm_setr_epi32(0x01010020, 0, 0, 0)), h1 = iv1;
        size_t at = n < 8 ? n : 8;
        __m512i m = _mm512_inserti64x4(_mm512_castsi256_si512(_mm256_loadu_si256((const __m256i*)head)),
                                       _mm256_maskz_loadu_epi32((__mmask8)((1u << at) - 1u), words), 1);
        uint64_t t = 64;
        for (;;) {
            const bool last = t >= bytes;
            const uint64_t count = last ? bytes : t;
            __m128i a = h0, b = h1, c = iv0, d = _mm_xor_si128(iv1, _mm_setr_epi32((int)count, (int)(count >> 32), last ? -1 : 0, 0));
#pragma GCC unroll 10
            for (int r = 0; r < 10; r++) {
                const __m512i w = _mm512_permutexvar_epi32(_mm512_load_si512(order.w[r]), m);
                half_round(a, b, c, d, _mm512_castsi512_si128(w), _mm512_extracti32x4_epi32(w, 1));
                a = _mm_shuffle_epi32(a, 0x93); d = _mm_shuffle_epi32(d, 0x4e); c = _mm_shuffle_epi32(c, 0x39);
                half_round(a, b, c, d, _mm512_extracti32x4_epi32(w, 2), _mm512_extracti32x4_epi32(w, 3));
                a = _mm_shuffle_epi32(a, 0x39); d = _mm_shuffle_epi32(d, 0x4e); c = _mm_shuffle_epi32(c, 0x93);
            }
            h0 = _mm_xor_si128(h0, _mm_xor_si128(a, c));
            h1 = _mm_xor_si128(h1, _mm_xor_si128(b, d));
            if (last) break;
            const size_t k = n - at < 16 ? n - at : 16;
            m = _mm512_maskz_loadu_epi32((__mmask16)((1u << k) - 1u), words + at);
            at += k;
            t += 64;
        }
        const __m256i w = _mm256_inserti128_si256(_mm256_castsi128_si256(h0), h1, 1), p = _mm256_set1_epi32((int)zk::P);
        const __m256i s = _mm256_add_epi32(_mm256_and_si256(w, p), _mm256_srli_epi32(w, 31));
        HashWords out;
        _mm256_storeu_si256((__m256i*)out.data(), _mm256_min_epu32(s, _mm256_sub_epi32(s, p)));
        return out;
    }
};
#undef B200_ROWS
#endif
inline HashWords hash_words_m31(const HashWords& head, const uint32_t* words, size_t n, uint64_t bytes) {
#if defined(__x86_64__)
    if (Blake2sRows::here()) return Blake2sRows::hash(head.data(), words, n, bytes);
#endif
    Blake2sState st;
    st.update_words(head.data(), 8);
    st.update_words(words, n);
    const uint8_t zeros[4] = {0, 0, 0, 0};
    st.update(zeros, (size_t)(bytes - 32 - 4 * n));
    return st.finalize_m31();
}

// Blake2sM31Channel.
class Channel {
  public:
    const HashWords& digest() const { return digest_; }
    void mix_root(const HashWords& root) { mix_u32s(root.data(), 8); }  // blake2_merkle.rs:53-58
    void mix_u32s(const uint32_t* data, size_t n) { set(hash_words_m31(digest_, data, n, 32 + 4 * (uint64_t)n)); }
    void mix_u64(uint64_t v) { uint32_t d[2] = {(uint32_t)v, (uint32_t)(v >> 32)}; mix_u32s(d, 2); }
    void mix_felts(const zk::qm31* f, size_t n) { mix_u32s((const uint32_t*)f, 4 * n); }
    void mix_felts(const std::vector<zk::qm31>& f) { mix_felts(f.data(), f.size()); }
    std::array<uint32_t, 8> draw_u32s() {  // the digest, the count of draws and a zero byte
        const uint32_t draws = n_draws_++;
        return hash_words_m31(digest_, &draws, 1, 37);
    }
    // channel/blake2s.rs:34-52: retry until all eight words are below 2p.
    std::array<uint32_t, 8> draw_base_felts() {
        for (;;) {
            auto u = draw_u32s();
            bool ok = true;
            for (auto x : u) ok = ok && x < 2 * zk::P;
            if (!ok) continue;
            for (auto& x : u) x = x >= zk::P ? x - zk::P : x;
            return u;
        }
    }
    zk::qm31 draw_secure_felt() {
        auto f = draw_base_felts();
        return {{f[0], f[1], f[2], f[3]}};
    }
    // H(POW_PREFIX, 12 zero bytes, digest, n_bits), channel/blake2s.rs:124-133
    HashWords pow_prefixed_digest(uint32_t n_bits) const {
        Blake2sState st;
        uint32_t head[4] = {0x12345678u, 0, 0, 0};
        st.update_words(head, 4);
        st.update_words(digest_.data(), 8);
        st.update_words(&n_bits, 1);
        return st.finalize_m31();
    }
    // The state as a device-resident copy of the channel holds it (digest, n_draws), and back.
    uint32_t n_draws() const { return n_draws_; }
    void set_state(const HashWords& d, uint32_t n_draws) { digest_ = d; n_draws_ = n_draws; }
  private:
    void set(const HashWords& d) { digest_ = d; n_draws_ = 0; }
    HashWords digest_{};
    uint32_t n_draws_ = 0;
};

// core/queries.rs:11-31
inline std::vector<size_t> draw_queries(Channel& ch, uint32_t log_domain_size, size_t n_queries) {
    std::vector<size_t> raw;
    uint32_t mask = (uint32_t)(((uint64_t)1 << log_domain_size) - 1);
    while (raw.size() < n_queries)
        for (auto w : ch.draw_u32s()) {
            raw.push_back(w & mask);
            if (raw.size() == n_queries) break;
        }
    return raw;
}

}  // namespace b200
