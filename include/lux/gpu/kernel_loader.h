/*
 * The directory of compiled-in kernels that a backend hands to the Lux GPU core (include/lux/gpu/kernel_loader.h:34-90
 * of the core): the layout only, for builds without a tree of the core (see backend_plugin.h beside this file).
 */
#ifndef LUX_GPU_KERNEL_LOADER_H
#define LUX_GPU_KERNEL_LOADER_H

#include <stddef.h>

#ifdef __cplusplus
extern "C" {
#endif

typedef enum { LUX_KERNEL_LANG_CUDA = 1 } LuxKernelLang; /* the one language this plugin's entries have */

typedef struct {
    const char *name, *entry_point;
    LuxKernelLang lang;
    const char* source;
    size_t source_len;
    const void* binary;
    size_t binary_len;
} LuxEmbeddedKernel;

typedef struct {
    const char* backend;
    const LuxEmbeddedKernel* kernels;
    size_t count;
} LuxKernelRegistry;

#ifdef __cplusplus
}
#endif
#endif /* LUX_GPU_KERNEL_LOADER_H */
