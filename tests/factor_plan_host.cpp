// factor_plan_host.cpp -- the host side of the sparse factorisation (tf_factor.cuh) without a GPU, linked
// against libtf_b200.so. tests/test_factor_plan.py builds it with g++ and reads what it prints.
#include <cinttypes>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "tf_factor.cuh"

int main(int argc, char** argv) {
    if (argc == 4 && !std::strcmp(argv[1], "span")) {  // of blocks [a, b)
        const tfb::FcSpan s = tfb::fc_block_span(std::atoi(argv[2]), std::atoi(argv[3]));
        std::printf("%" PRId64 " %" PRId64 "\n", s.begin, s.end);
        return 0;
    }
    return 2;
}
