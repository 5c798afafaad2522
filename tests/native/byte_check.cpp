// byte_over (dl_math.cuh) against the division it stands for, over every byte value, signed and
// unsigned, and both divisors. Built and run by tests/test_byte_over.py.
#include <cstdio>
#include <cstring>

#include "dl_math.cuh"

int main() {
    int bad = 0;
    const float divisors[2] = {127.0f, 255.0f};
    for (float n : divisors)
        for (int i = -128; i < 256; ++i) {
            const float got = dl::byte_over((float)i, n, 1.0f / n), want = (float)i / n;
            if (std::memcmp(&got, &want, 4)) ++bad;
        }
    std::printf("mismatches %d\n", bad);
    return bad ? 1 : 0;
}
