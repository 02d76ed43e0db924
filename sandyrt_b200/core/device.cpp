#include "device.h"

#include <algorithm>
#include <cstring>

#include "kernels.h"
#include "weights.h"

namespace sandy {

void cuda_check(cudaError_t e, const char* what) {
    if (e != cudaSuccess) throw KernelError(std::string(what) + ": " + cudaGetErrorString(e));
}

DeviceBuffer::DeviceBuffer(size_t bytes) : bytes_(bytes) {
    cuda_check(cudaMalloc(&ptr_, std::max<size_t>(bytes, 16)), "allocating device memory");
}
DeviceBuffer DeviceBuffer::if_there_is_room(size_t bytes) {
    DeviceBuffer b;
    const cudaError_t e = cudaMalloc(&b.ptr_, std::max<size_t>(bytes, 16));
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();             // answered here: no launch behind this one reports it
        b.ptr_ = nullptr;
        return b;
    }
    cuda_check(e, "allocating device memory");
    b.bytes_ = bytes;
    return b;
}
DeviceBuffer::~DeviceBuffer() {
    if (ptr_) cudaFree(ptr_);
}
DeviceBuffer& DeviceBuffer::operator=(DeviceBuffer&& o) noexcept {
    if (this != &o) {
        if (ptr_) cudaFree(ptr_);
        ptr_ = o.ptr_;
        bytes_ = o.bytes_;
        o.ptr_ = nullptr;
        o.bytes_ = 0;
    }
    return *this;
}

PinnedBuffer::PinnedBuffer(size_t bytes) : bytes_(bytes) {
    cuda_check(cudaMallocHost(&ptr_, std::max<size_t>(bytes, 16)), "allocating pinned host memory");
    std::memset(ptr_, 0, std::max<size_t>(bytes, 16));
}
PinnedBuffer::~PinnedBuffer() {
    if (ptr_) cudaFreeHost(ptr_);
}
PinnedBuffer& PinnedBuffer::operator=(PinnedBuffer&& o) noexcept {
    if (this != &o) {
        if (ptr_) cudaFreeHost(ptr_);
        ptr_ = o.ptr_;
        bytes_ = o.bytes_;
        o.ptr_ = nullptr;
        o.bytes_ = 0;
    }
    return *this;
}

thread_local TransposeStage* TransposeStage::current_ = nullptr;

DeviceWeight to_device(const HostTensor& t, DType compute, bool keep_32bit, bool transpose, bool as_rows) {
    int64_t rows = 1, cols = t.numel();
    if (t.shape.size() >= 2 && as_rows) {
        rows = t.shape[0];
        cols = rows ? t.numel() / rows : 0;
    }
    DeviceWeight w;
    const void* src = nullptr;
    std::vector<float> f32;
    std::vector<uint16_t> b16;
    std::vector<int32_t> i32;
    DType dt;
    if (!store_dtype_is_float(t.dtype)) {
        dt = DType::I32;
        i32 = to_i32(t);
        src = i32.data();
    } else if (compute == DType::F32 || (keep_32bit && t.dtype == StoreDType::F32)) {
        dt = DType::F32;
        if (t.dtype == StoreDType::F32) src = t.data;
        else { f32 = to_f32(t); src = f32.data(); }
    } else {
        dt = DType::BF16;
        if (t.dtype == StoreDType::BF16) src = t.data;
        else { b16 = to_bf16_bits(t); src = b16.data(); }
    }
    const size_t esz = dtype_size(dt);
    if (transpose && t.shape.size() != 2) throw ValueError("only a matrix can be transposed");
    const size_t bytes = (size_t)t.numel() * esz;
    w.buffer = std::make_shared<DeviceBuffer>(bytes);
    if (transpose && t.numel()) {
        // turned on the device: on the host it costs as much as reading the file (28 M floats: 60 to 200 ms)
        TransposeStage own, *stage = own.outer() ? own.outer() : &own;
        void* raw = stage->room(bytes);
        cuda_check(cudaMemcpy(raw, src, bytes, cudaMemcpyHostToDevice), "copying a weight to the device");
        const int code = SANDY_KERNEL(elementwise, sandy_transpose)(raw, w.buffer->get(), rows, cols, (int)esz, nullptr);
        if (code) throw KernelError("transposing a weight: code " + std::to_string(code));
        cuda_check(cudaStreamSynchronize(nullptr), "transposing a weight");
    } else if (t.numel()) {
        cuda_check(cudaMemcpy(w.buffer->get(), src, bytes, cudaMemcpyHostToDevice), "copying a weight to the device");
    }
    if (transpose) std::swap(rows, cols);
    w.view.data = w.buffer->get();
    w.view.dtype = dt;
    w.view.rows = rows;
    w.view.cols = cols;
    w.view.ld = cols;
    return w;
}

Tensor Workspace::get(const std::string& name, int64_t rows, int64_t cols, DType dtype) {
    Tensor t;
    t.data = raw(name + ":" + dtype_name(dtype), (size_t)(rows * cols) * dtype_size(dtype));
    t.dtype = dtype;
    t.rows = rows;
    t.cols = cols;
    t.ld = cols;
    return t;
}

std::vector<Tensor> Workspace::get_together(const std::string& name, int64_t rows, const std::vector<std::pair<int64_t, DType>>& cols) {
    std::vector<size_t> at;
    size_t bytes = 0;
    for (const auto& [n, dtype] : cols) {
        at.push_back(bytes);
        bytes += ((size_t)(rows * n) * dtype_size(dtype) + 255) / 256 * 256;
    }
    char* base = (char*)raw(name, bytes);
    std::vector<Tensor> out(cols.size());
    for (size_t i = 0; i < cols.size(); i++) {
        out[i].data = base + at[i];
        out[i].dtype = cols[i].second;
        out[i].rows = rows;
        out[i].cols = out[i].ld = cols[i].first;
    }
    return out;
}

void* Workspace::raw(const std::string& name, size_t bytes) {
    auto key = std::make_pair(name, 0);
    auto it = bufs_.find(key);
    if (it == bufs_.end() || it->second.bytes() < bytes) {
        // grow in steps, so that a slowly growing step does not move the buffer every time
        size_t want = std::max<size_t>(bytes, 256);
        if (it != bufs_.end()) want = std::max(want, it->second.bytes() + it->second.bytes() / 2);
        DeviceBuffer larger = DeviceBuffer::if_there_is_room(want);
        if (!larger.get()) {
            give_back();
            larger = DeviceBuffer(want);
        }
        bufs_[key] = std::move(larger);
        version_++;
        it = bufs_.find(key);
    }
    return it->second.get();
}

void* Workspace::spare(const std::string& name, size_t bytes) {
    Spare& s = spares_[name];
    if (s.buffer.get() && s.buffer.bytes() >= bytes) return s.buffer.get();
    if (bytes >= s.refused) return nullptr;
    if (s.buffer.get()) version_++;
    s.buffer = DeviceBuffer();          // nothing in it outlives the call it was asked for
    s.buffer = DeviceBuffer::if_there_is_room(bytes);
    if (s.buffer.get()) version_++;
    else s.refused = bytes;
    return s.buffer.get();
}

bool Workspace::give_back() {
    bool any = false;
    for (auto& [name, s] : spares_)
        if (s.buffer.get()) {
            s.refused = std::min(s.refused, s.buffer.bytes());
            s.buffer = DeviceBuffer();
            any = true;
        }
    if (any) version_++;
    return any;
}

}  // namespace sandy
