// modal_batch.h -- batches of linear constant-coefficient instances on the modal kernel (modal_batch.cu).
#pragma once
#include <cuda_runtime.h>

#include <vector>

struct bosss_handle;

namespace bosss {

struct ModalBatch;
// *out stays null (no error) where an instance does not qualify
int modal_batch_create(const std::vector<bosss_handle*>& hs, const long long* dom_off, const long long* cod_off,
                       ModalBatch** out);
void modal_batch_destroy(ModalBatch* m);
int modal_batch_run(const ModalBatch* m, int mode, double alpha, double beta, const double* U, const double* V,
                    double* out, cudaStream_t s);

}  // namespace bosss
