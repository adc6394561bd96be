// The Mersenne Twister MT19937 (Matsumoto and Nishimura, ACM TOMACS 8(1), 1998) with the state layout and the
// double conversion of numpy's legacy RandomState, so that the submitter thread can draw the coordinate noise
// of a shuffled training pass from numpy's global stream without holding the interpreter lock.  (Drawn by
// numpy in a Python submitter, the noise and the hand-over cost 0.6 ms a batch of 1024 molecules against
// 0.15 ms of GPU work.)  A block of 624 words is advanced in three loops whose iterations are independent of
// one another, so that the compiler vectorises them, with AVX2 where the machine has it: 41 thousand values, the noise of
// 1024 molecules, which batches draw one after the other, 70 -> 47 us.  (Not with FMA: that would round once less.)
#pragma once

#include <cstdint>

#if defined(__x86_64__) && defined(__GNUC__) && !defined(__clang__)
#define ANI_HOST_SIMD __attribute__((target_clones("avx2", "default")))
#else
#define ANI_HOST_SIMD
#endif

namespace ani {

class Mt19937 {
  public:
    static constexpr int kN = 624, kM = 397;
    void set(const uint32_t* key, int pos)
    {
        for (int i = 0; i < kN; i++) key_[i] = key[i];
        pos_ = pos;
        temper();
    }
    void get(uint32_t* key, int* pos) const
    {
        for (int i = 0; i < kN; i++) key[i] = key_[i];
        *pos = pos_;
    }
    // n doubles of low + range * u, u uniform in [0, 1) with 53 bits from two words each.
    ANI_HOST_SIMD void uniform(double* out, long long n, double low, double range)
    {
        while (n > 0) {
            if (pos_ >= kN) refill();
            const int pairs = (kN - pos_) / 2;
            if (pairs == 0) {      // the two words of this value lie in different blocks
                const uint32_t a = word_[pos_];
                refill();
                *out++ = low + range * to_double(a, word_[pos_++]);
                n--;
                continue;
            }
            const int take = n < pairs ? (int)n : pairs;
            const uint32_t* w = word_ + pos_;
            for (int i = 0; i < take; i++) out[i] = low + range * to_double(w[2 * i], w[2 * i + 1]);
            out += take;
            n -= take;
            pos_ += 2 * take;
        }
    }

  private:
    static double to_double(uint32_t a, uint32_t b)
    {
        return ((double)(int32_t)(a >> 5) * 67108864.0 + (double)(int32_t)(b >> 6)) * (1.0 / 9007199254740992.0);
    }
    static uint32_t twist(uint32_t u, uint32_t v)
    {
        const uint32_t y = (u & 0x80000000u) | (v & 0x7fffffffu);
        return (y >> 1) ^ ((0u - (v & 1u)) & 0x9908b0dfu);
    }
    ANI_HOST_SIMD void refill()
    {
        for (int i = 0; i < kN - kM; i++) key_[i] = key_[i + kM] ^ twist(key_[i], key_[i + 1]);
        for (int i = kN - kM; i < kN - 1; i++) key_[i] = key_[i + kM - kN] ^ twist(key_[i], key_[i + 1]);
        key_[kN - 1] = key_[kM - 1] ^ twist(key_[kN - 1], key_[0]);
        pos_ = 0;
        temper();
    }
    ANI_HOST_SIMD void temper()
    {
        for (int i = 0; i < kN; i++) {
            uint32_t y = key_[i];
            y ^= y >> 11;
            y ^= (y << 7) & 0x9d2c5680u;
            y ^= (y << 15) & 0xefc60000u;
            word_[i] = y ^ (y >> 18);
        }
    }
    uint32_t key_[kN] = {}, word_[kN] = {};
    int pos_ = kN;
};

}  // namespace ani
