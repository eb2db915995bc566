// tpd_kernels.h — host-side launch interface of the splatting kernels.
// Plain C++ (no CUDA syntax) so the engine and the C ABI can include it.
#pragma once
#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

namespace tpd {

struct ViewConst;
struct Splat;

// Per-engine control block in device memory.
struct FrameCtl {
    uint32_t status;         // kStatus* bits, cleared at frame start
    uint32_t tag;            // launch tag, advanced once per frame / call
    uint32_t total_keys;     // K, written by the tile-count scan (0xFFFFFFFF: 2^31 keys or more)
    uint32_t visible;        // (view, Gaussian) pairs with a non-empty tile rect
    uint32_t ticket[32];     // partition tickets, cleared at frame start
    uint32_t sort_hist[8][256];   // digit counts of the key sort, by 8-bit digit position
    uint32_t depth_hist[8][256];  // digit counts of the depth sort, by 8-bit digit position
    uint32_t debug[4];       // site, index, bound of the first failed index guard
    uint32_t depth_count;    // (view, Gaussian) items with a non-empty tile rect: those the depth sort keeps
    // depth-sort passes skipped because their digit was the same for every
    // key (the order stays in the pass's input buffer): when odd, the later
    // passes swap their buffers and the sorted items are in the other one
    uint32_t depth_skips;
    uint32_t tile_order_done;  // CTAs of the tile order that have finished (reset by the last)
    uint32_t total_strips;     // column strips of the visible items, written by the tile-count scan
    uint32_t tile_hist[128];    // tiles by class of their walk length (tile_class), counted by the blend
    uint32_t tile_cursor[128];  // tiles of each class that the tile order has placed (0 at rest)
    uint32_t list_class[32];    // tiles by class of their list length, as launch_list_classes places them
};
constexpr uint32_t kListClasses = 16;

// Entity matrices: rows 0..2 of view*model and rows 0..3 of projview*model.
constexpr int kEntityMatFloats = 28;

// Ticket slots and look-back tag slots (tag = ctl->tag * 32 + slot).
constexpr int kTicketPreprocess = 0;
constexpr int kTicketScan = 1;
constexpr int kTicketBlend = 2;           // tile queue of a persistent blend launch
constexpr int kTicketBlendBackward = 3;   // tile queue of a persistent adjoint launch (reset by tile order)
constexpr int kTicketKeySortBase = 8;     // + 8-bit digit position
constexpr int kTicketDepthSortBase = 16;  // + 8-bit digit position
constexpr uint32_t kTagScan = 0;
constexpr uint32_t kTagKeySort = 1;       // + digit position
constexpr uint32_t kTagDepthSort = 16;    // + digit position

struct PreprocessArgs {
    const float* recs;        // n x 60 floats (240-byte records)
    uint32_t n;
    const uint32_t* ent_idx;  // per-Gaussian entity index or nullptr (entity 0)
    const float* ent_mats;    // n_views x n_ent x kEntityMatFloats
    uint32_t n_ent;
    const ViewConst* views;   // device, n_views
    uint32_t n_views;         // <= kMaxViews
    uint32_t sh_degree;
    uint32_t band3_compat;
    Splat* splats;            // n_views x n (view-major)
    // depth-sort input (nullptr: not written): item = v * n + i,
    // key = (v << 32) | bits(viewZ), or (v << 32) | 0xFFFFFFFF when culled
    uint64_t* depth_keys;
    uint32_t* depth_items;
    uint32_t depth_key_bits;  // 32 + bits of (n_views - 1); its digit histograms go to ctl->depth_hist
    FrameCtl* ctl;
};

constexpr uint32_t kMaxViews = 256;

// Kernel set-up that must happen once per device (a shared-memory opt-in, an
// occupancy query): calls init() the first time it is asked for on the
// current device and returns that result on every later call there.
// Thread-safe; keyed by (device, init).
int device_once(int (*init)());

// The test hook of the standalone scans (tpd_test_set_never_publish).
uint32_t test_never_publish_standalone();

// Clears tickets, histograms and status of ctl and advances its tag; computes
// entity matrices for n_views x n_ent (transforms nullptr -> identity).
void launch_frame_begin(FrameCtl* ctl, const float* transforms, uint32_t n_ent, const ViewConst* views,
                        uint32_t n_views, float* ent_mats, cudaStream_t s);
void launch_preprocess(const PreprocessArgs& a, int num_sms, cudaStream_t s);

// Splats per partition of the standalone scan.
constexpr uint32_t kScanTilesPart = 4096;
constexpr size_t scan_tiles_desc_entries(uint64_t n) { return size_t((n + kScanTilesPart - 1) / kScanTilesPart); }
// Standalone exclusive scan of Splat.tiles (prefix.slang) into offsets, total
// into *total, device status into *status. Clears everything it starts from:
// desc (scan_tiles_desc_entries(n) descriptors) and ctl's ticket.
void launch_scan_tiles(const Splat* splats, uint32_t n, uint32_t* offsets, uint32_t* total, uint64_t* desc,
                       FrameCtl* ctl, uint32_t* status, uint32_t spin_limit, uint32_t never_publish, cudaStream_t s);

// Items (view, Gaussian) in depth order per partition of the depth-order
// scan: its look-back descriptors number n_items / kKeygenPart + 2.
constexpr uint32_t kKeygenPart = 1024;

// The tile counts of the ctl->depth_count (view, Gaussian) items in depth
// order (items[r] = v * n + i < n_items) scanned into exclusive key offsets
// offsets[r] (prefix.slang), then keygen.slang's key duplication: keys
// (tile_base + tile) << 32 | bits(viewZ) with vals = Gaussian index. The
// items come in depth order, so only the tile id of each key is written
// (tiles[], u32): the depth half of a key is the depth of its value's splat
// (launch_materialize_keys). K goes to ctl->total_keys and the non-empty
// count to ctl->visible; more keys than the capacity, or 2^31 of them, flag the
// frame (kStatusKeyOverflow) and none are written. Also presets ranges (2 x n_tiles
// u32) to (0xFFFFFFFF, 0) for the key sort's last pass.
struct KeygenArgs {
    const Splat* splats;
    const uint32_t* items;        // where the depth sort leaves the order with no pass skipped
    const uint32_t* items_other;  // the other buffer, which holds it when ctl->depth_skips is odd
    uint32_t n_items;             // views x n
    uint32_t n;                   // Gaussians per view
    const ViewConst* views;
    uint32_t* offsets;            // n_items
    uint4* item_info;             // n_items: scratch between the two kernels
    uint32_t* part_first;         // ceil(capacity / 4096): scratch between the two kernels
    uint32_t* tiles;              // capacity, 16-byte aligned
    uint32_t* vals;               // capacity, 16-byte aligned
    uint32_t capacity;
    uint32_t* ranges;
    uint32_t n_tiles;
    uint32_t tile_bits;           // tile ids are below 2^tile_bits
    uint64_t* desc;               // look-back descriptors (tag ctl->tag * 32 + kTagScan), never cleared
    // the key sort's counted work area: the first pass is counted and its
    // offsets are ready afterwards (SortPlan.precounted); nullptr: the digit
    // counts of the tile ids go to ctl->sort_hist instead
    uint32_t* counted_work;
    // strips (launch_strip_sort follows, see takes_strips): one view; column
    // strips are written instead of keys, and their columns counted
    bool strips;
    uint64_t* strip_desc;         // look-back descriptors of the strip counts, as desc
    FrameCtl* ctl;
    uint32_t spin_limit;
    uint32_t never_publish;
};
void launch_keygen(const KeygenArgs& a, int num_sms, cudaStream_t s);

// The key sort by strips. A frame's keys are the tiles of its rectangles; a
// strip is one column of a rectangle, and there are several times fewer of them
// than keys. launch_keygen (KeygenArgs.strips) writes them in depth order; here
// they are sorted by column, then expanded into their keys while those are
// sorted by row: the keys themselves are moved once. The sorted values are in
// vals, and the ranges written, as by the last pass of launch_sort.
struct StripSort {
    uint32_t *strips, *vals, *strips_alt, *vals_alt;  // capacity each; the strips are in the first two
    uint32_t* starts;      // capacity: scratch
    uint32_t* part_first;  // ceil(capacity / 4096): scratch
    uint32_t capacity;
    uint32_t* work;        // the counted work area; the columns are counted
    uint32_t* ranges;
    uint32_t n_tiles;
    uint32_t gx;           // the image's tile columns
    FrameCtl* ctl;
    uint32_t max_parts() const { return capacity > 4096u ? (capacity + 4095u) / 4096u : 1u; }
};
bool takes_strips(uint32_t n_views, uint32_t gx, uint32_t gy);  // whether a frame's key sort does (gx x gy tiles)
void launch_strip_sort(const StripSort& a, cudaStream_t s);

// keys[i] = tile << 32 | bits(viewZ of splat vals[i] in the tile's view) for
// the slots i < min(ctl->total_keys, capacity) of every tile's range: the
// 64-bit (tile | depth) keys of a frame, from its tile ranges and sorted values
// (read-back only).
void launch_materialize_keys(const uint32_t* ranges, uint32_t n_tiles, const uint32_t* vals, const Splat* splats,
                             uint32_t n, const uint32_t* tile_view, uint32_t capacity, const FrameCtl* ctl,
                             uint64_t* keys, cudaStream_t s);

// Onesweep LSD radix sort of (key, val) pairs on key bits [first_bit, key_bits),
// first_bit a multiple of 8. K = min(ctl->total_keys, capacity). hist: the
// [8][256] digit counts by digit position (hist_ready: already filled, else a
// histogram kernel builds them); tickets ctl->ticket[ticket_base + position];
// look-back tags ctl->tag * 32 + tag_base + position. Result in (keys, vals)
// for an even pass count, else in (keys_alt, vals_alt); returns true for *_alt.
// desc: sort_desc_entries(capacity, items) descriptors (tagged, never cleared).
size_t sort_desc_entries(uint32_t capacity, uint32_t items = 16);
// Keys per thread of the 256-thread onesweep passes over n 64-bit pairs, 4, 8
// or 16: fewer where 4096-key partitions would leave SMs idle.
uint32_t sort_items_for(uint32_t n);
uint32_t sort_items_limit(uint32_t items);  // the most pairs sorted with that many
uint32_t sort_pass_count(uint32_t key_bits);
struct SortPlan {
    uint32_t first_bit = 0;
    uint32_t key_bits = 64;
    uint32_t (*hist)[256] = nullptr;
    bool hist_ready = false;
    uint32_t ticket_base = kTicketKeySortBase;
    uint32_t tag_base = kTagKeySort;
    int ctas_per_sm = 2;
    uint32_t items = 16;               // keys per thread: 16 (4096-key partitions), 8 or 4
    uint32_t threads = 256;            // 512: 4096-key partitions as 512 threads x 8 keys (items unused)
    uint32_t* ranges = nullptr;        // key sort: the last pass also writes the tile ranges (preset by keygen)
    uint32_t n_tiles = 0;
    uint32_t fixed_count = 0;          // nonzero: sort this many pairs, else min(ctl->total_keys, capacity)
    // a frame whose keys overflowed the capacity sorts nothing (none were
    // written); it is rendered again
    bool skip_on_overflow = false;
    // depth sort: the first pass drops the keys whose low 32 bits are
    // 0xFFFFFFFF (culled items) and keeps ctl->depth_count, which the later
    // passes sort; a later pass whose digit is the same for every key copies
    bool compact_culled = false;
    cudaEvent_t after_hist = nullptr;  // recorded between the histogram and the first pass
    // non-null, 32-bit keys: counted passes (every partition's digit offsets
    // counted and scanned beforehand, no look-back; plain pass kinds only) using this work
    // area of sort_counted_work_words(capacity) u32, zeroed once (every launch
    // leaves its arrival counts at zero). With ranges, the last pass writes
    // them and the values, not the keys
    uint32_t* counted_work = nullptr;
    // counted passes: the first pass's digit offsets are already in
    // counted_work, put there by the kernel that wrote the keys right before
    // this sort (launch_keygen)
    bool precounted = false;
};
size_t sort_counted_work_words(uint32_t capacity);
// Digit width of the counted passes over keys of key_bits bits: 9 where that
// takes fewer passes than 8.
uint32_t counted_digit_bits(uint32_t key_bits);
bool launch_sort(uint64_t* keys, uint32_t* vals, uint64_t* keys_alt, uint32_t* vals_alt, uint32_t capacity,
                 const SortPlan& plan, uint64_t* desc, FrameCtl* ctl, uint32_t spin_limit, int num_sms,
                 cudaStream_t s);
// The same for 32-bit keys (the frame's tile ids).
bool launch_sort(uint32_t* keys, uint32_t* vals, uint32_t* keys_alt, uint32_t* vals_alt, uint32_t capacity,
                 const SortPlan& plan, uint64_t* desc, FrameCtl* ctl, uint32_t spin_limit, int num_sms,
                 cudaStream_t s);
// Few pairs: the whole sort as one launch (sort_small.cu). The depth form
// writes the first ctl->depth_count items (their position in keys) in (view,
// depth) order; the plain one sorts (keys, vals) on the low key_bits bits into
// (keys_out, vals_out), other buffers than the inputs, and clears ctl->status.
constexpr uint32_t kSmallSortMax = 12288;
void launch_small_depth_sort(const uint64_t* keys, uint32_t* items_out, uint32_t n, uint32_t key_bits, FrameCtl* ctl,
                             cudaStream_t s);
void launch_small_sort(const uint64_t* keys, const uint32_t* vals, uint64_t* keys_out, uint32_t* vals_out, uint32_t n,
                       uint32_t key_bits, FrameCtl* ctl, cudaStream_t s);

// Clears status, histograms and tickets, sets total_keys and advances the tag
// (standalone stage calls).
void launch_sort_begin(FrameCtl* ctl, uint32_t total, cudaStream_t s);


// The tiles by class of their list length (octaves, longest first), for the
// blend: class c's tiles fill buckets[c n_tiles ..), ctl->list_class[c] of them.
void launch_list_classes(const uint32_t* ranges, uint32_t n_tiles, FrameCtl* ctl, uint32_t* buckets, cudaStream_t s);
// Whether a frame of n_tiles blends in that order.
bool blend_takes_list_order(uint32_t n_tiles, int num_sms);

struct BlendArgs {
    const Splat* splats;      // n_views x n (view-major)
    uint32_t n;               // Gaussians per view
    FrameCtl* ctl;            // K = min(ctl->total_keys, capacity); frames with a fatal status are skipped
    uint32_t capacity;
    const uint32_t* vals;
    uint32_t* ranges;         // 2 x n_tiles (global tile ids); an empty tile's (0xFFFFFFFF, 0) is rewritten to (0, 0)
    const ViewConst* views;   // device, n_views entries
    const uint32_t* tile_view;  // per global tile: view index (nullptr: single view 0)
    uint32_t n_tiles;
    const uint32_t* list_buckets;  // nullable: CTAs take the tiles in launch_list_classes' order
    float* image;             // HWC float3 per view, packed per view at image_offset[view]
    const uint64_t* image_offset;  // per view pixel offset (nullptr: 0)
    // per pixel: final transmittance and list entries up to the last
    // contributor (the adjoint's inputs); both null: not tracked
    float* final_T;
    uint32_t* n_contrib;
    // with them: per tile, the list entries up to its last contributor, whose
    // classes are counted in ctl->tile_hist (for launch_tile_order); the top bit
    // is set where a pixel's colour is infinite or close to it
    uint32_t* tile_len;
    // nullable: the image also as RGBA8 UNORM (alpha 255), packed like image
    // (launch_pack_rgba8's conversion), written with it
    uint32_t* rgba;
};
// Launch settings of the blend and its adjoint: list entries per staged
// round (forward 64 / 128 / 256, adjoint 32 / 64 / 128) and the form of the
// launch: one CTA per tile, or persistent CTAs (SMs x resident CTAs) taking
// (view, tile) items from a queue in FrameCtl. None of them changes a result.
struct BlendLaunch {
    uint32_t round = 128;
    uint32_t backward_round = 64;
    bool persistent = false;
    int num_sms = 148;
};
void launch_blend(const BlendArgs& a, const BlendLaunch& l, cudaStream_t s);

// RGBA8 UNORM pack of an HWC float3 image (alpha 1), the reference's target format.
void launch_pack_rgba8(const float* rgb, uint32_t* rgba, size_t pixels, cudaStream_t s);

// ---- backward
struct BlendBackwardArgs {
    const Splat* splats;      // n_views x n (view-major)
    uint32_t n;               // Gaussians per view
    FrameCtl* ctl;
    uint32_t capacity;
    const uint32_t* vals;
    const uint32_t* ranges;
    const ViewConst* views;
    const uint32_t* tile_view;
    uint32_t n_tiles;
    const uint64_t* image_offset;
    const float* final_T;
    const uint32_t* n_contrib;
    const float* dL_dimage;   // HWC float3
    float* g2d;               // n x kG2DStride (px, py, conic.xyz, opacity, rgb, 3 pad), accumulated
    uint64_t g2d_view_stride; // floats between views' g2d (n * kG2DStride)
    const uint32_t* tile_len;    // as the blend left it
    const uint32_t* tile_order;  // nullable: CTA b differentiates tile tile_order[b] (launch_tile_order)
};
void launch_blend_backward(const BlendBackwardArgs& a, const BlendLaunch& l, cudaStream_t s);

// order[0 .. n_tiles): the tiles by decreasing walk length (classes of a
// quarter octave; any order within a class), so the longest walks of the
// adjoint start first and no SM is left with one at the end. tile_len and
// ctl->tile_hist as the last blend that kept the adjoint's inputs left them.
// Also resets the adjoint's tile queue.
void launch_tile_order(const uint32_t* tile_len, uint32_t n_tiles, FrameCtl* ctl, uint32_t* order, cudaStream_t s);

// Per-splat gradient record of the blend adjoint: 9 used floats padded to 12
// (48 B), so it is accumulated with three 16-byte vector atomics.
constexpr uint32_t kG2DStride = 12;

struct PreprocessBackwardArgs {
    const float* recs;
    uint32_t n;
    const uint32_t* ent_idx;
    const float* ent_mats;    // per view: n_ent x 28, view-major
    uint32_t n_ent;
    const ViewConst* views;   // device
    uint32_t n_views;
    uint32_t sh_degree;
    uint32_t band3_compat;
    const Splat* splats;      // per view n splats, view-major
    const float* g2d;         // per view n x kG2DStride, view-major
    float* g_means;           // n x 3
    float* g_log_scales;      // n x 3
    float* g_quats;           // n x 4
    float* g_logits;          // n
    float* g_sh;              // n x 48
};
void launch_preprocess_backward(const PreprocessBackwardArgs& a, cudaStream_t s);

// Raw parameters -> 240-byte records: opacity = sigmoid(logit), scale = exp(log_scale)
// with modifier 1, quaternion and SH copied as given.
void launch_pack_records(const float* means, const float* log_scales, const float* quats, const float* logits,
                         const float* sh, uint32_t n, float* recs, cudaStream_t s);

}  // namespace tpd
