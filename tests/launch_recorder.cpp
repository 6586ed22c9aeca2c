// A CUDA runtime that launches nothing: it stands in for libcudart under the library's own host code (see
// test_launch_sequence.py) and writes down every kernel launch, one line each:
//   <mangled kernel name> grid=<x> cluster=<x> cooperative=<0|1> programmatic=<0|1> stream=<handle> status=<address>
// (status: the word into which the kernels of the dense MLP report a wait that ran out; 0 for others).
// "Device" memory is host memory that nothing reads; events, copies and attributes succeed.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <map>
#include <string>

namespace {
std::map<const void*, std::string>& names() {
  static std::map<const void*, std::string> table;
  return table;
}
std::string log_text;
int current_device = 0, current_sms = 148;
struct Pending {
  dim3 grid, block;
  size_t shared;
  cudaStream_t stream;
} pending;

// DensePairParams::status of dense_gemm_pair.cu, GemmParams::status of gv_gemm_parts.cuh and FewParams::status of dense_few_rows.cu, by their places.
size_t status_of(const std::string& name, void** arguments) {
  if (name.find("dense_fp8_pair_kernel") != std::string::npos) return static_cast<size_t*>(arguments[2])[1];
  if (name.find("grouped_nvfp4_gemm_kernel") != std::string::npos) return static_cast<size_t*>(arguments[3])[13];
  if (name.find("dense_few_") != std::string::npos) return static_cast<size_t*>(arguments[1])[5];
  return 0;
}

void record(const void* function, unsigned grid, unsigned cluster, bool cooperative, bool programmatic, cudaStream_t stream,
            void** arguments) {
  char line[512];
  std::snprintf(line, sizeof(line), "%s grid=%u cluster=%u cooperative=%d programmatic=%d stream=%zu status=%zu\n",
                names()[function].c_str(), grid, cluster, cooperative, programmatic, reinterpret_cast<size_t>(stream),
                status_of(names()[function], arguments));
  log_text += line;
}

CUresult encode_tiled_stub(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                           const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                           CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  return CUDA_SUCCESS;
}
}  // namespace

extern "C" {

const char* recorder_take_log() {
  static std::string taken;
  taken.swap(log_text);
  log_text.clear();
  return taken.c_str();
}

// From now on the current device is this one, of so many SMs.
void recorder_set_device(int device, int sms) {
  current_device = device;
  current_sms = sms;
}

void** __cudaRegisterFatBinary(void*) {
  static void* handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) {
  names()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shared, cudaStream_t stream) {
  pending = {grid, block, shared, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* shared, void* stream) {
  *grid = pending.grid;
  *block = pending.block;
  *shared = pending.shared;
  *static_cast<cudaStream_t*>(stream) = pending.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* function, dim3 grid, dim3, void** arguments, size_t, cudaStream_t stream) {
  record(function, grid.x, 1, false, false, stream, arguments);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* config, const void* function, void** arguments) {
  unsigned cluster = 1;
  bool cooperative = false, programmatic = false;
  for (unsigned i = 0; i < config->numAttrs; ++i) {
    const cudaLaunchAttribute& a = config->attrs[i];
    if (a.id == cudaLaunchAttributeClusterDimension) cluster = a.val.clusterDim.x;
    if (a.id == cudaLaunchAttributeCooperative) cooperative = a.val.cooperative != 0;
    if (a.id == cudaLaunchAttributeProgrammaticStreamSerialization)
      programmatic = a.val.programmaticStreamSerializationAllowed != 0;
  }
  record(function, config->gridDim.x, cluster, cooperative, programmatic, config->stream, arguments);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "recorded"; }

cudaError_t cudaMalloc(void** pointer, size_t bytes) {
  *pointer = std::aligned_alloc(512, (bytes + 511) / 512 * 512);
  return *pointer ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaMallocAsync(void** pointer, size_t bytes, cudaStream_t) { return cudaMalloc(pointer, bytes); }
cudaError_t cudaFree(void* pointer) {
  std::free(pointer);
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* pointer, cudaStream_t) { return cudaFree(pointer); }
cudaError_t cudaMemcpy(void*, const void*, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemset(void*, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** pointer, const void* symbol) {
  *pointer = const_cast<void*>(symbol);
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* device) {
  *device = current_device;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* value, cudaDeviceAttr attribute, int) {
  *value = attribute == cudaDevAttrComputeCapabilityMajor ? 10 : attribute == cudaDevAttrMultiProcessorCount ? current_sms : 0;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* properties, int) {
  *properties = cudaDeviceProp{};
  properties->major = 10;
  properties->multiProcessorCount = current_sms;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** function, unsigned long long, cudaDriverEntryPointQueryResult* result) {
  *function = reinterpret_cast<void*>(&encode_tiled_stub);
  if (result) *result = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* stream, unsigned) {
  *stream = nullptr;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* status) {
  *status = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* event, unsigned) {
  *event = nullptr;
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }

}  // extern "C"
