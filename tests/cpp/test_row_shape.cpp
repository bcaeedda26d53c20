// row_shape (ciflow_gb300/csrc/row_shape.h): "<rows> <elements> <fp64> <kind>" per line of
// the input, "<lanes> <chunks>" per line of the output.
#include "../../ciflow_gb300/csrc/row_shape.h"

#include <cstdio>

int main() {
    long long n, nnz;
    int fp64, kind;
    while (std::scanf("%lld %lld %d %d", &n, &nnz, &fp64, &kind) == 4) {
        const cigpu::RowShape s = cigpu::row_shape(n, nnz, fp64 != 0, (cigpu::RowKind)kind);
        std::printf("%d %d\n", s.lanes, s.chunks);
    }
    return 0;
}
