// Test helper for tests/test_friction_scale.py: reads pairs (bound, q2) of float or double from a binary
// file (int bits, int n, then the values) and writes friction_scale of each.
#include <cstdio>
#include <vector>
#include "pe_math.cuh"

template <class R> static int run(FILE* in, FILE* out, int n) {
    std::vector<R> v((size_t)2 * n), r(n);
    if (std::fread(v.data(), sizeof(R), v.size(), in) != v.size()) return 1;
    for (int i = 0; i < n; i++) r[i] = pe::friction_scale(v[2 * i], v[2 * i + 1]);
    return std::fwrite(r.data(), sizeof(R), n, out) == (size_t)n ? 0 : 1;
}

int main(int argc, char** argv) {
    if (argc < 3) return 2;
    FILE *in = std::fopen(argv[1], "rb"), *out = std::fopen(argv[2], "wb");
    int h[2];
    if (!in || !out || std::fread(h, 4, 2, in) != 2) return 2;
    const int rc = h[0] == 32 ? run<float>(in, out, h[1]) : run<double>(in, out, h[1]);
    std::fclose(out);
    return rc;
}
