// The cuBLAS entry points that the gradient loads, for tests/grad_create/harness.cu: GEMMs report the bytes that
// each operand spans (column-major) and do nothing.
#include <cstddef>
#include <cstdint>

extern "C" {
void harness_operand(const void *p, size_t bytes);

int cublasCreate_v2(void **h) {
   static int handle;
   *h = &handle;
   return 0;
}
int cublasDestroy_v2(void *) { return 0; }
int cublasSetStream_v2(void *, void *) { return 0; }
int cublasSetWorkspace_v2(void *, void *ws, size_t n) {
   harness_operand(ws, n);
   return 0;
}
int cublasGemmEx(void *, int ta, int tb, int m, int n, int k, const void *, const void *A, int, int lda, const void *B, int,
                 int ldb, const void *, void *C, int, int ldc, int, int) {
   auto span = [](int rows, int cols, int ld) { return 4 * ((size_t)ld * (cols - 1) + rows); };
   harness_operand(A, ta ? span(k, m, lda) : span(m, k, lda));
   harness_operand(B, tb ? span(n, k, ldb) : span(k, n, ldb));
   harness_operand(C, span(m, n, ldc));
   return 0;
}
}
