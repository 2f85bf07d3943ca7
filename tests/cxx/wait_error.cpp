// Reads of results throw what a kernel has reported through the engine's error flag, once.
#include <cuPoly/arithmetic/polynomial.h>
#include <cuPoly/cuda/cudaengine.h>
#include <cupoly_b200.h>

#include <cstdio>
#include <exception>

int main() {
  CUDAEngine::init_bfv(2, 3, 4096, 256);
  int rc = 0;
  {
    Context ctx;
    poly_t a;
    poly_init(&ctx, &a);
    poly_set_coeff(&ctx, &a, 3, NTL::ZZ(7));
    poly_add(&ctx, &a, &a, &a);
    for (int v = 0; v < 2; ++v) {
      if (cp_wait_test(CUDAEngine::handle(), ctx.get_stream()) != CP_OK) return 2;
      try {
        if (v == 0)
          poly_get_coeff(&ctx, &a, 3);
        else
          poly_export_residues(&ctx, &a);
        rc = 1;
      } catch (const std::exception& e) {
        std::printf("%s\n", e.what());
      }
    }
    std::printf("%ld\n", NTL::conv<long>(poly_get_coeff(&ctx, &a, 3)));
    poly_free(&ctx, &a);
  }
  CUDAEngine::destroy();
  return rc;
}
