// noalloc.cu - a render entry point that allocates no memory.
//
// Some callers cannot call cudaMalloc: a host application that already owns all GPU
// memory through its own pool or arena, a plugin loaded into a process whose allocator
// must not be bypassed, or code running while a CUDA graph is being recorded elsewhere.
// vxr_render_frame_noalloc renders one frame for them from device buffers they already
// own (the world grid, its bricks and the light list) into an image buffer they own.
// Everything else the frame needs - G-buffer, seeds, both reservoir planes, the hit
// list, the shadow-ray queue, the uber cells' tables, the brick boxes of a world of up to
// 32,768 bricks, the per-light table, the counters and the device error word - lives in one file-scope
// __device__ array of fixed size, which every GPU that loads this library holds until
// the process exits (VXR_NOALLOC_SCRATCH_BYTES = 10,518,784 bytes, 10.0 MiB).
//
// The stage kernels are the ones the view path launches; only the buffers differ.
#include <cstring>
#include <mutex>
#include <string>

#include <cuda_runtime.h>

#include "internal.hpp"
#include "kernels.hpp"
#include "view.hpp"

namespace {

constexpr size_t kMaxPx = VXR_NOALLOC_MAX_PIXELS;
constexpr size_t kMaxLights = VXR_NOALLOC_MAX_LIGHTS;
// layout (byte offsets, every region 256-byte aligned)
constexpr size_t kOffVd = 0;                                   // uint2 [kMaxPx]
constexpr size_t kOffSeed = kOffVd + 8 * kMaxPx;               // uint32 [kMaxPx]
constexpr size_t kOffCA = kOffSeed + 4 * kMaxPx;               // uint4 [kMaxPx]
constexpr size_t kOffCB = kOffCA + 16 * kMaxPx;                // float4 [kMaxPx]
constexpr size_t kOffHA = kOffCB + 16 * kMaxPx;                // uint4 [kMaxPx]
constexpr size_t kOffHB = kOffHA + 16 * kMaxPx;                // float4 [kMaxPx]
constexpr size_t kOffUber = kOffHB + 16 * kMaxPx;              // uint8 [32^3]
constexpr size_t kOffGeom = kOffUber + 32 * 32 * 32;           // float4 [kMaxLights]
constexpr size_t kOffEmit = kOffGeom + 16 * kMaxLights;        // float4 [kMaxLights]
constexpr size_t kOffTables = kOffEmit + 16 * kMaxLights;      // 16 * kMaxLights bytes: the uber cells' tables, brick boxes
constexpr size_t kOffHits = kOffTables + 16 * kMaxLights;      // uint32 [kMaxPx] hit list
constexpr size_t kOffQA = kOffHits + 4 * kMaxPx;               // float4 [kMaxPx] shadow requests
constexpr size_t kOffQB = kOffQA + 16 * kMaxPx;                // float4 [kMaxPx]
constexpr size_t kOffErr = kOffQB + 16 * kMaxPx;               // uint32 error word, then the work-list counters
constexpr size_t kScratchBytes = kOffErr + 256;
static_assert(kScratchBytes == VXR_NOALLOC_SCRATCH_BYTES, "scratch size must match the header");
static_assert(kOffSeed % 256 == 0 && kOffCA % 256 == 0 && kOffUber % 256 == 0 && kOffGeom % 256 == 0 &&
                  kOffHits % 256 == 0 && kOffQA % 256 == 0 && kOffErr % 256 == 0,
              "scratch regions must stay 256-byte aligned");
static_assert(16 * kMaxLights >= (16 + 8) * 32 * 32 * 32, "the uber cells' tables must fit their region");
// bricks whose boxes (two words each) fit what they leave of it
constexpr size_t kMaxBoxes = (16 * kMaxLights - (16 + 8) * 32 * 32 * 32) / 8;

__device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

// Host-side address of g_noalloc_scratch per device. The symbol's name in host code is
// only a host stand-in, so the device address is looked up once per device with
// cudaGetSymbolAddress while that device is current.
constexpr int kMaxDevices = 64;
unsigned char* g_scratch_ptr[kMaxDevices] = {};
std::mutex g_scratch_mutex;

int scratch_for_current_device(unsigned char** out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return vxr::set_error(VXR_E_NODEVICE, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
    if (dev < 0 || dev >= kMaxDevices) return vxr::set_error(VXR_E_INVALID, "vxr_render_frame_noalloc: device index >= 64");
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_ptr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p)
            return vxr::set_error(VXR_E_CUDA, std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
        g_scratch_ptr[dev] = (unsigned char*)p;
    }
    *out = g_scratch_ptr[dev];
    return VXR_OK;
}

}  // namespace

#define CUN(call, what)                                                                                     \
    do {                                                                                                    \
        cudaError_t e_ = (call);                                                                            \
        if (e_ != cudaSuccess) return vxr::set_error(VXR_E_CUDA, std::string(what) + ": " + cudaGetErrorString(e_)); \
    } while (0)

extern "C" int vxr_render_frame_noalloc(const uint32_t* grid, const uint32_t* bricks, uint32_t nbricks,
                                        const vxr_light* lights, uint32_t nlights, uint32_t light_model,
                                        const vxr_frame_consts* k, float* out_rgba, void* stream) {
    VXR_CHECK_ARG(grid && bricks && k && out_rgba && (lights || nlights == 0), "vxr_render_frame_noalloc: null argument");
    VXR_CHECK_ARG(light_model == VXR_LIGHTS_AREA || light_model == VXR_LIGHTS_POINT,
                  "vxr_render_frame_noalloc: unknown light model");
    VXR_CHECK_ARG(k->width >= 1 && k->height >= 1, "vxr_render_frame_noalloc: empty frame");
    if ((size_t)k->width * k->height > kMaxPx)
        return vxr::set_error(VXR_E_INVALID, "vxr_render_frame_noalloc: " + std::to_string(k->width) + "x" +
                                                 std::to_string(k->height) + " exceeds the fixed scratch of " +
                                                 std::to_string(kMaxPx) + " pixels");
    if (nlights > kMaxLights)
        return vxr::set_error(VXR_E_INVALID, "vxr_render_frame_noalloc: " + std::to_string(nlights) +
                                                 " lights exceed the fixed scratch of " + std::to_string(kMaxLights));
    VXR_CHECK_ARG(k->numberOfLights == nlights, "vxr_render_frame_noalloc: numberOfLights differs from nlights");
    VXR_CHECK_ARG(k->spatialRadius >= 1, "vxr_render_frame_noalloc: spatialRadius must be >= 1");
    VXR_CHECK_ARG(nbricks >= 1, "vxr_render_frame_noalloc: nbricks must be >= 1");

    unsigned char* s = nullptr;
    if (int r = scratch_for_current_device(&s)) return r;
    cudaStream_t st = (cudaStream_t)stream;
    uint32_t* err = (uint32_t*)(s + kOffErr);
    CUN(cudaMemsetAsync(err, 0, kScratchBytes - kOffErr, st), "clear error word and counters");

    // derive the light table and the uber cells' tables in scratch; the latter's kernel also
    // checks the grid and raises kBadGrid, which keeps the pixel stages from reading bricks
    // through a bad one and from writing the image: one wait, at the end (with a wait for the
    // check in between, and light records widened by a kernel of their own, 242 us instead of 223)
    float4* geom = (float4*)(s + kOffGeom);
    float4* emit = (float4*)(s + kOffEmit);
    static_assert(sizeof(vxr_light) == 12, "three words a light");
    vxr::launch_build_light_table(reinterpret_cast<const uint32_t*>(lights), 3, nlights, geom, emit, st);
    uint4* ucell0 = (uint4*)(s + kOffTables);
    unsigned long long* ucell = (unsigned long long*)(ucell0 + 32 * 32 * 32);
    // and, behind them, when the world's bricks are few enough, the boxes of their opaque and of
    // their non-zero voxels. Reading every brick once (3,734 bricks 3 us, 16,122 some 8) pays
    // for itself: a frame in us without and with boxes, 256 x 144 of 3,734 bricks 255 and 239,
    // 200 x 120 of 16,122 337 and 330, 160 x 90 of 15,547 with 30,000 emitters 514 and 392.
    uint32_t* box = nbricks <= kMaxBoxes ? (uint32_t*)(ucell + 32 * 32 * 32) : nullptr;
    uint32_t* box0 = box ? box + nbricks : nullptr;
    if (box) vxr::launch_build_brick_boxes(bricks, nullptr, nbricks, box, box0, nullptr, nullptr, st);
    vxr::launch_build_cells(grid, box, box0, s + kOffUber, ucell, ucell0, nullptr, nullptr, nbricks, err, st);
    CUN(cudaGetLastError(), "world kernels");

    vxr::dev::World w;
    w.grid = grid;
    w.uber = s + kOffUber;
    w.bricks = bricks;
    w.bbox = box;   // null: rays walk every brick they meet
    w.bbox0 = box0;
    w.ubox0 = nullptr;
    w.ucell = ucell;
    w.ucell0 = ucell0;
    w.lgeom = geom;
    w.lemit = emit;
    w.nlights = nlights;

    // a single frame: no temporal history is read (the scratch keeps the previous
    // call's contents, which may belong to another world or camera)
    vxr::dev::Frame f = vxr::dev_frame(*k);
    f.restirtemporalframe = 0;
    f.temporal = 0;
    f.accumulate = 0;
    f.sky = nullptr;

    vxr::ViewBuffers b;
    b.vd[0] = (uint2*)(s + kOffVd);
    b.vd[1] = (uint2*)(s + kOffVd);          // previous G-buffer: never read without temporal reuse
    b.seed = (uint32_t*)(s + kOffSeed);
    b.cA = (uint4*)(s + kOffCA);
    b.cB = (float4*)(s + kOffCB);
    b.hA = (uint4*)(s + kOffHA);
    b.hB = (float4*)(s + kOffHB);
    b.frame = (float4*)out_rgba;
    b.accum = (float4*)out_rgba;             // unused: shading runs without the accumulate fusion
    b.err = err;
    b.hits = (uint32_t*)(s + kOffHits);
    b.qA = (float4*)(s + kOffQA);
    b.qB = (float4*)(s + kOffQB);
    b.counters = (uint32_t*)(s + kOffErr + 64);
    const bool point = light_model == VXR_LIGHTS_POINT;
    const vxr::Tuning sh;
    vxr::BatchDev bd = vxr::single_batch(w, f, b, 0, point, sh);
    bd.lists = 1;
    bd.cleared = 1;
    bd.halt = err;
    const int variant = point ? 1 : 0;
    vxr::launch_batch_albedo(bd, variant, st);
    vxr::launch_batch_candidates(bd, variant, nullptr, st);
    vxr::launch_batch_spatial(bd, variant, st);
    vxr::launch_batch_shade(bd, variant, st);
    CUN(cudaGetLastError(), "stage kernels");
    uint32_t herr = 0;
    CUN(cudaMemcpyAsync(&herr, err, sizeof(uint32_t), cudaMemcpyDeviceToHost, st), "read error word");
    CUN(cudaStreamSynchronize(st), "vxr_render_frame_noalloc");
    if (herr & vxr::kBadGrid)
        return vxr::set_error(VXR_E_INVALID, "vxr_render_frame_noalloc: grid references a brick >= nbricks");
    if (herr) return vxr::set_error(VXR_E_DEVICE, "vxr_render_frame_noalloc: " + vxr::device_flags_message(herr));
    return VXR_OK;
}
