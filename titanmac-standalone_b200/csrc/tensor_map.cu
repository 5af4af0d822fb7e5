#include "tensor_map.cuh"

#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>

#include "tmw_common.cuh"

namespace tmw {
namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
    });
    return fn;
}

// Encoded maps are kept per host thread, keyed by everything that goes into them: a caller that runs the same buffers
// again pays for the driver call once.  One slot per hash value - a whole model's weights (four maps per layer) have to
// find room beside the activations', and a search through a list of that many is as long as the driver call.
struct MapKey {
    int64_t v[11];
    bool operator==(const MapKey& o) const { return std::memcmp(v, o.v, sizeof(v)) == 0; }
};
struct Slot {
    MapKey key;
    CUtensorMap map;
    bool used = false;
};
constexpr int kSlots = 1024;

Slot& slot_of(const MapKey& key) {
    static thread_local std::unique_ptr<Slot[]> slots;
    if (!slots) slots.reset(new Slot[kSlots]);
    uint64_t h = 1469598103934665603ull;
    for (int64_t x : key.v) h = (h ^ (uint64_t)x) * 1099511628211ull, h ^= h >> 29;
    return slots[h % kSlots];
}

bool encode(CUtensorMap* map, int dtype, int rank, const void* base, const cuuint64_t* dims, const cuuint64_t* strides,
            const cuuint32_t* box, CUtensorMapSwizzle swizzle) {
    EncodeTiledFn fn = encode_fn();
    if (fn == nullptr) return false;
    const cuuint32_t elem_strides[4] = {1, 1, 1, 1};
    const CUtensorMapDataType dt = dtype == TMW_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    const CUresult r = fn(map, dt, rank, const_cast<void*>(base), dims, strides, box, elem_strides,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r == CUDA_SUCCESS) return true;
    char text[96];
    snprintf(text, sizeof(text), "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
    set_error_text(text);
    return false;
}

}  // namespace

bool make_map_2d(CUtensorMap* map, const void* base, int dtype, int rows, int cols, int64_t ld, int box_rows, int box_cols,
                 CUtensorMapSwizzle swizzle) {
    const MapKey key{{2, (int64_t)(uintptr_t)base, ld, dtype, rows, cols, box_rows, box_cols, (int64_t)swizzle, 0, 0}};
    Slot& s = slot_of(key);
    if (!s.used || !(s.key == key)) {
        const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
        const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
        const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
        s.used = encode(&s.map, dtype, 2, base, dims, strides, box, swizzle);
        if (!s.used) return false;
        s.key = key;
    }
    *map = s.map;
    return true;
}

MapStrides map_strides(int batch, int heads, int rows, int dh, const int64_t stride[3]) {
    MapStrides m;
    m.row = rows > 1 ? stride[2] : dh;
    m.head = heads > 1 ? stride[1] : m.row * rows;
    const int64_t inner_span = m.head * heads > m.row * rows ? m.head * heads : m.row * rows;
    m.batch = batch > 1 ? stride[0] : inner_span;
    m.heads_first = m.head < m.row;
    const int64_t limit = ((int64_t)1 << 40) / 2;
    m.ok = m.row > 0 && m.head > 0 && m.batch > 0 && m.row < limit && m.head < limit && m.batch < limit &&
           m.row % 8 == 0 && m.head % 8 == 0 && m.batch % 8 == 0;
    return m;
}

bool make_map_4d(CUtensorMap* map, const void* base, int dtype, int batch, int heads, int rows, int dh, const MapStrides& m,
                 int box_rows) {
    const MapKey key{{4, (int64_t)(uintptr_t)base, m.row, m.head, m.batch, dtype, batch, heads, rows, dh, box_rows}};
    Slot& s = slot_of(key);
    if (!s.used || !(s.key == key)) {
        cuuint64_t dims[4], strides[3];
        cuuint32_t box[4];
        dims[0] = (cuuint64_t)dh;
        box[0] = 64;
        if (m.heads_first) {
            dims[1] = (cuuint64_t)heads; strides[0] = (cuuint64_t)m.head * 2; box[1] = 1;
            dims[2] = (cuuint64_t)rows;  strides[1] = (cuuint64_t)m.row * 2;  box[2] = (cuuint32_t)box_rows;
        } else {
            dims[1] = (cuuint64_t)rows;  strides[0] = (cuuint64_t)m.row * 2;  box[1] = (cuuint32_t)box_rows;
            dims[2] = (cuuint64_t)heads; strides[1] = (cuuint64_t)m.head * 2; box[2] = 1;
        }
        dims[3] = (cuuint64_t)batch;
        strides[2] = (cuuint64_t)m.batch * 2;
        box[3] = 1;
        s.used = encode(&s.map, dtype, 4, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
        if (!s.used) return false;
        s.key = key;
    }
    *map = s.map;
    return true;
}

}  // namespace tmw
