// The CUDA runtime calls that the library makes, for tests of its host code
// without a GPU: memory is the host's, kernels are not run, and every launch,
// function attribute, allocation and synchronisation is recorded.  A launch is
// refused, as the runtime refuses it, where it asks for more dynamic shared
// memory than its kernel's attribute allows, or where the test says so
// (fake_refuse); a refused launch leaves a capture that it is part of valid.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

namespace {
struct Launch {
	std::string name;
	unsigned grid, block;
	size_t smem;
	int programmatic;
};
constexpr int SMEM_DEFAULT = 48 * 1024, SMEM_OPTIN = 232448;
std::mutex mu;
std::map<const void*, std::string> names;
std::map<std::string, std::vector<int>> smem_attr;  // every value set, in order
std::vector<Launch> launches;                       // accepted ones, captured ones included
std::string refuse;
long long nalloc = 0, nlive = 0, nsync = 0, nrefused = 0, ngraph = 0;
cudaError_t last = cudaSuccess;
thread_local struct {
	dim3 grid, block;
	size_t smem;
	cudaStream_t stream;
} pushed;

cudaError_t record(cudaError_t e) {
	if (e != cudaSuccess) last = e;
	return e;
}
cudaError_t launch(const void* fn, dim3 grid, dim3 block, size_t smem, int programmatic) {
	std::lock_guard<std::mutex> lock(mu);
	const std::string& name = names[fn];
	const auto a = smem_attr.find(name);
	const int most = a == smem_attr.end() ? SMEM_DEFAULT : a->second.back();
	if ((!refuse.empty() && name.find(refuse) != std::string::npos) || smem > (size_t)most || block.x > 1024) {
		nrefused++;
		return record(cudaErrorInvalidValue);
	}
	launches.push_back({name, grid.x, block.x, smem, programmatic});
	return cudaSuccess;
}
}  // namespace

extern "C" {
void** __cudaRegisterFatBinary(void*) {
	static void* handle;
	return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) {
	names[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
	pushed = {grid, block, smem, stream};
	return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
	*grid = pushed.grid;
	*block = pushed.block;
	*smem = pushed.smem;
	*static_cast<cudaStream_t*>(stream) = pushed.stream;
	return cudaSuccess;
}

cudaError_t cudaLaunchKernel(const void* fn, dim3 grid, dim3 block, void**, size_t smem, cudaStream_t) {
	return launch(fn, grid, block, smem, 0);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void**) {
	int programmatic = 0;
	for (unsigned i = 0; i < c->numAttrs; ++i)
		if (c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization)
			programmatic |= c->attrs[i].val.programmaticStreamSerializationAllowed;
	return launch(fn, c->gridDim, c->blockDim, c->dynamicSmemBytes, programmatic);
}
cudaError_t cudaFuncSetAttribute(const void* fn, cudaFuncAttribute attr, int value) {
	std::lock_guard<std::mutex> lock(mu);
	if (attr != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
	if (value > SMEM_OPTIN) return record(cudaErrorInvalidValue);
	smem_attr[names[fn]].push_back(value);
	return cudaSuccess;
}
cudaError_t cudaGetLastError() {
	const cudaError_t e = last;
	last = cudaSuccess;
	return e;
}
const char* cudaGetErrorString(cudaError_t) { return "refused by the test"; }

cudaError_t cudaMalloc(void** p, size_t n) {
	nalloc++;
	nlive++;
	*p = std::calloc(n, 1);
	return *p ? cudaSuccess : record(cudaErrorMemoryAllocation);
}
cudaError_t cudaFree(void* p) {
	if (p) nlive--;
	std::free(p);
	return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
	std::memmove(d, s, n);
	return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
	return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
	std::memset(d, v, n);
	return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }

cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) {
	*d = 0;
	return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
	*v = a == cudaDevAttrMultiProcessorCount ? 148 : (a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? SMEM_OPTIN : 0);
	return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult* q) {
	*p = nullptr;
	if (q) *q = cudaDriverEntryPointSymbolNotFound;
	return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
	*p = nullptr;
	return cudaErrorInvalidSymbol;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
	*s = reinterpret_cast<cudaStream_t>(std::malloc(1));
	return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
	std::free(s);
	return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
	nsync++;
	return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
	*e = reinterpret_cast<cudaEvent_t>(std::malloc(1));
	return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
	std::free(e);
	return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
	*ms = 1.0f;
	return cudaSuccess;
}

cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
	*g = reinterpret_cast<cudaGraph_t>(std::malloc(1));
	return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* ge, cudaGraph_t, unsigned long long) {
	*ge = reinterpret_cast<cudaGraphExec_t>(std::malloc(1));
	return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
	ngraph++;
	return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
	std::free(g);
	return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t g) {
	std::free(g);
	return cudaSuccess;
}

// ------------------------------------------------------- the tests' side
void fake_reset() {
	launches.clear();
	refuse.clear();
	last = cudaSuccess;
	nalloc = nsync = nrefused = ngraph = 0;
}
// Refuses every launch of a kernel whose name contains `part` ("": none).
void fake_refuse(const char* part) { refuse = part; }
// [allocations, live allocations, stream synchronisations, refused launches, graph launches]
void fake_counts(long long* out) {
	const long long v[] = {nalloc, nlive, nsync, nrefused, ngraph};
	std::memcpy(out, v, sizeof v);
}
long long fake_launches() { return (long long)launches.size(); }
const char* fake_launch(long long i, long long* out) {
	const Launch& l = launches[i];
	const long long v[] = {l.grid, l.block, (long long)l.smem, l.programmatic};
	std::memcpy(out, v, sizeof v);
	return l.name.c_str();
}
// Values a kernel's shared-memory attribute has been set to: how many different ones, over all kernels the most.
long long fake_most_smem_settings() {
	size_t most = 0;
	for (const auto& a : smem_attr) {
		std::map<int, int> seen;
		for (int v : a.second) seen[v] = 1;
		most = std::max(most, seen.size());
	}
	return (long long)most;
}
}
