// Device-resident octree topology (dtopo.cu): the reference's per-level hash tables, their
// compaction and the refinement / coarsening / ghost-spawning / cell-type steps run on the GPU,
// bit-exact with the host Topology and the reference (tile order = hash-slot order).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

namespace cirrus {

// One hash slot on the device: tile coordinates and meta = tile-memory id | type << 24, or -1
// when empty.
struct __align__(16) DSlot {
    int x, y, z, meta;
};

class DevTopology {
public:
    DevTopology(int num_layers, const uint32_t* log2_hash, double h0);
    ~DevTopology();
    DevTopology(const DevTopology&) = delete;
    DevTopology& operator=(const DevTopology&) = delete;

    int num_layers() const { return num_layers_; }
    double h0() const { return h0_; }
    int max_level() const { return max_level_; }
    const uint32_t* log2_hash() const { return log2_.data(); }
    int num_tiles() const;

    // setTileHost with blank tiles, in the given order (one level per call)
    int set_tiles(int level, const int32_t* xyz, const uint8_t* types, int n);
    int compress_and_sync();                          // compressHost + syncHostAndDevice
    int spawn_ghost_tiles();                          // SpawnGhostTiles
    // RefineLeafsOneStep / CoarsenStep with level targets from dense per-level masks:
    // refine: target = level + (mask != 0); coarsen: target = level - (mask != 0)
    int refine_leafs_one_step(const std::vector<const uint8_t*>& masks, const std::vector<int>& dims, std::vector<int>* counts);
    int iterative_refine(const std::vector<const uint8_t*>& masks, const std::vector<int>& dims);
    int coarsen_step(const std::vector<const uint8_t*>& masks, const std::vector<int>& dims, std::vector<int>* deleted);
    int set_cell_types(const uint8_t* host_ct);       // all tiles, all-tiles order
    int calc_cell_types_from_leafs();                 // CalcCellTypesFromLeafs

    // all-tiles order exports (host arrays)
    int tiles(int32_t* out5) const;
    int hash_slots(int32_t* out) const;
    int cell_types(uint8_t* out) const;
    int statuses(int32_t* out) const;
    std::string last_error;

private:
    // device memory that only grows; the first `cap` bytes are part of d_base_ (owned: its own allocation)
    struct Buffer {
        void* p = nullptr;
        size_t cap = 0;
        bool owned = false;
    };
    int ensure_mem(int extra);
    int renumber_mem();
    int grow(Buffer* b, size_t bytes) const;
    int read_ctl(int* ctl);
    int refine_step(std::vector<int>* counts);
    int upload_masks(const std::vector<const uint8_t*>& masks, const std::vector<int>& dims);
    template <class Launch> int export_with(size_t bytes, void* host, Launch&& launch) const;

    int num_layers_;
    double h0_;
    int max_level_ = -1;
    std::vector<uint32_t> log2_;
    int device_ = -1;
    unsigned long long context_ = 0;    // id of the primary context it was made in; 0: another kind
    size_t base_bytes_ = 0;
    void* d_base_ = nullptr;            // one allocation: the tables, d_ctl_ and what is between, the buffers' first sizes
    std::vector<DSlot*> live_, snap_;   // per level: the edited table and the synced copy
    std::vector<DSlot*> arr_;           // per level: compacted snapshot (hash-slot order)
    std::vector<int> count_;            // per level: tiles in arr_
    bool stale_ = false;                // the live tables were edited since the last compaction (also by a step that failed)
    int* d_claims_ = nullptr;           // per slot of every level: the insertion claim
    size_t claim_slots_ = 0;
    int4* d_chunks_ = nullptr;          // compaction chunks: level, chunk, the level's first chunk
    int* d_chunk_count_ = nullptr;
    int n_chunks_ = 0;
    DSlot** d_live_ = nullptr;          // device arrays of the per-level pointers
    DSlot** d_snap_ = nullptr;
    DSlot** d_arr_ = nullptr;
    int** d_claim_ = nullptr;
    uint8_t** d_masks_ = nullptr;       // level-target masks (in d_mask_buf_)
    uint32_t* d_log2_ = nullptr;
    int* d_mask_dims_ = nullptr;
    int* d_ctl_ = nullptr;              // counters read back after each pass of a step
    Buffer mask_buf_;
    Buffer scratch_;                    // lists of refined tiles, ghost candidates, clusters
    Buffer found_;                      // per child of the refined tiles: its slot and the parent's memory
    int32_t* status_ = nullptr;         // per tile memory
    uint8_t* ctype_ = nullptr;          // 512 per tile memory
    bool mem_owned_ = false;            // status_ and ctype_ are allocations of their own
    int mem_count_ = 0, mem_cap_ = 0;
    mutable Buffer export_;             // staging of the exports
    mutable std::mutex export_lock_;
};

}  // namespace cirrus
