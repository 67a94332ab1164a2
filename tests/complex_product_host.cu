// complex_product_host.cu -- cmul and cmul_conj of utr_public_gb300/csrc/fft_line.cuh,
// compiled for the host, on the pairs (a, b) in argv[1]; a b, then a conj(b), of each
// to argv[2].  TEST ONLY: lets the CPU tests bound their roundings without a GPU.
#include <cstdio>
#include <vector>

#include "fft_line.cuh"

int main(int argc, char **argv)
{
    if (argc < 3) return 2;
    std::vector<float2> out;
    float2 ab[2];
    FILE *f = fopen(argv[1], "rb");
    if (!f) return 3;
    while (fread(ab, sizeof(float2), 2, f) == 2) {
        out.push_back(msk::cmul(ab[0], ab[1]));
        out.push_back(msk::cmul_conj(ab[0], ab[1]));
    }
    fclose(f);
    f = fopen(argv[2], "wb");
    if (!f || fwrite(out.data(), sizeof(float2), out.size(), f) != out.size()) return 4;
    fclose(f);
    return 0;
}
