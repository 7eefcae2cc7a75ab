/*
 * The binary interface of a Lux GPU backend plugin, ABI version 2, as this plugin needs it to be compiled: handle
 * types, enum values, the 64-slot table and the descriptor (include/lux/gpu/backend_plugin.h:30-445 of the Lux GPU
 * core).  The build takes the core's own header where a tree of it lies beside this repository; this declaration of
 * the same layout is what it is compiled against otherwise.  The slots this plugin never fills are untyped here.
 * plugin.cu asserts the sizes and offsets that a core relies on.
 */
#ifndef LUX_GPU_BACKEND_PLUGIN_H
#define LUX_GPU_BACKEND_PLUGIN_H

#include <stdbool.h>
#include <stddef.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

#define LUX_GPU_BACKEND_ABI_VERSION 2
#define LUX_GPU_BACKEND_EXPORT __attribute__((visibility("default")))

typedef struct LuxBackendContext LuxBackendContext;
typedef struct LuxBackendBuffer LuxBackendBuffer;
typedef struct LuxBackendKernel LuxBackendKernel;

typedef enum {
    LUX_DTYPE_FLOAT32, LUX_DTYPE_FLOAT16, LUX_DTYPE_BFLOAT16, LUX_DTYPE_INT32,
    LUX_DTYPE_INT64, LUX_DTYPE_UINT32, LUX_DTYPE_UINT64, LUX_DTYPE_BOOL
} LuxBackendDtype;

typedef enum {
    LUX_BACKEND_OK, LUX_BACKEND_ERROR_INVALID_ARGUMENT, LUX_BACKEND_ERROR_OUT_OF_MEMORY,
    LUX_BACKEND_ERROR_NOT_SUPPORTED, LUX_BACKEND_ERROR_DEVICE_LOST, LUX_BACKEND_ERROR_INTERNAL
} LuxBackendError;

/* capability bits; a bit whose position only the core's header fixes is not announced (0) */
#define LUX_CAP_TENSOR_OPS 0x1u
#define LUX_CAP_MATMUL 0x2u
#define LUX_CAP_NTT 0u
#define LUX_CAP_CUSTOM_KERNELS 0u

typedef struct {
    const char *name, *vendor;
    uint64_t memory_total, memory_available;
    int compute_units, max_workgroup_size;
    bool is_discrete, is_unified_memory;
} LuxBackendDeviceInfo;

#define LUX_CTX LuxBackendContext*
#define LUX_BUF LuxBackendBuffer*
typedef LuxBackendError (*lux_op_map_fn)(LUX_CTX, LUX_BUF in, LUX_BUF out, size_t n);
typedef LuxBackendError (*lux_op_pair_fn)(LUX_CTX, LUX_BUF a, LUX_BUF b, LUX_BUF out, size_t n);
typedef LuxBackendError (*lux_op_rows_fn)(LUX_CTX, LUX_BUF in, LUX_BUF out, size_t outer, size_t inner);
typedef LuxBackendError (*lux_op_ntt_fn)(LUX_CTX, uint64_t* data, size_t n, uint64_t modulus);

typedef struct lux_gpu_backend_vtbl {
    LUX_CTX (*create_context)(int device_index);
    void (*destroy_context)(LUX_CTX);
    LuxBackendError (*get_device_count)(int* count);
    LuxBackendError (*get_device_info)(LUX_CTX, LuxBackendDeviceInfo* info);
    LuxBackendError (*sync)(LUX_CTX);

    LUX_BUF (*buffer_alloc)(LUX_CTX, size_t bytes);
    LUX_BUF (*buffer_alloc_with_data)(LUX_CTX, const void* data, size_t bytes);
    void (*buffer_free)(LUX_CTX, LUX_BUF);
    LuxBackendError (*buffer_copy_to_host)(LUX_CTX, LUX_BUF, void* dst, size_t bytes);
    LuxBackendError (*buffer_copy_from_host)(LUX_CTX, LUX_BUF, const void* src, size_t bytes);
    void* (*buffer_get_host_ptr)(LUX_CTX, LUX_BUF);

    LuxBackendKernel* (*kernel_load)(LUX_CTX, const char* source, const char* entry_point);
    LuxBackendKernel* (*kernel_load_binary)(LUX_CTX, const void* binary, size_t bytes, const char* entry_point);
    void (*kernel_destroy)(LUX_CTX, LuxBackendKernel*);
    LuxBackendError (*kernel_dispatch)(LUX_CTX, LuxBackendKernel*, uint32_t grid_x, uint32_t grid_y, uint32_t grid_z,
                                       uint32_t block_x, uint32_t block_y, uint32_t block_z, LUX_BUF* buffers, int num_buffers);

    lux_op_pair_fn op_add_f32, op_sub_f32, op_mul_f32, op_div_f32;
    LuxBackendError (*op_matmul_f32)(LUX_CTX, LUX_BUF a, LUX_BUF b, LUX_BUF out, int M, int K, int N);
    LuxBackendError (*op_transpose_f32)(LUX_CTX, LUX_BUF in, LUX_BUF out, int rows, int cols);
    lux_op_map_fn op_reduce_sum_f32, op_reduce_max_f32, op_reduce_min_f32, op_reduce_mean_f32;
    lux_op_rows_fn op_reduce_sum_axis_f32, op_reduce_max_axis_f32, op_softmax_f32, op_log_softmax_f32;
    lux_op_map_fn op_exp_f32, op_log_f32, op_sqrt_f32, op_neg_f32, op_abs_f32, op_tanh_f32, op_sigmoid_f32, op_relu_f32,
        op_gelu_f32, op_copy_f32;
    LuxBackendError (*op_layer_norm_f32)(LUX_CTX, LUX_BUF in, LUX_BUF out, LUX_BUF gamma, LUX_BUF beta, size_t batch, size_t dim,
                                         float eps);
    LuxBackendError (*op_rms_norm_f32)(LUX_CTX, LUX_BUF in, LUX_BUF out, LUX_BUF weight, size_t batch, size_t dim, float eps);
    lux_op_ntt_fn op_ntt_forward, op_ntt_inverse; /* data: host memory, transformed in place */

    void *op_msm, *op_poly_mul, *op_tfhe_bootstrap, *op_tfhe_keyswitch, *op_blind_rotate, *op_sample_extract, *op_sample_ntt,
        *op_poseidon2_hash, *op_blake3_hash, *op_bls12_381_add, *op_bls12_381_mul, *op_bls12_381_pairing, *op_bn254_add,
        *op_bn254_mul, *op_kzg_commit, *op_kzg_open, *op_kzg_verify;
    void* _reserved[4];
} lux_gpu_backend_vtbl;
#undef LUX_CTX
#undef LUX_BUF

typedef struct {
    uint32_t abi_version;
    const char *backend_name, *backend_version;
    uint32_t capabilities;
    const lux_gpu_backend_vtbl* vtbl;
} lux_gpu_backend_desc;

#ifdef __cplusplus
}
#endif
#endif /* LUX_GPU_BACKEND_PLUGIN_H */
