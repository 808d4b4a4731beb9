// cafe_internal.h -- declarations shared by the translation units of libcafe_b200 (not installed).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "cafe_types.h"

struct CafeSortDesc;   // radix_sort.cuh


#define CAFE_MAX_DIM 128      // widest embedding row the scatter workspace is sized for
#define CAFE_CHUNK 32         // sorted lookups reduced by one thread group in the scatter
#define CAFE_CHUNK_SMALL 8            // ... in calls of
#define CAFE_CHUNK_SMALL_MOST 131072  // at most so many lookups

struct CafeSketchView {
    const CafeMainBucket* main;
    int n1, n2, lim, cap;
};

// Device buffers of the embedding path, sized once per handle for `cap` lookups.
struct CafeEmbedWorkspace {
    int cap = 0;
    float* norm = nullptr;       // [cap] gradient norm per lookup
    float* imp = nullptr;        // [cap] importance per lookup
    float* totals = nullptr;     // [CAFE_MAX_SEGMENTS] sum of norms per field
    int32_t* mask = nullptr;     // [cap] newly-hot flag per lookup
    int32_t* post_row = nullptr; // [cap] hot row after the lookup's own call
    uint32_t* key = nullptr;                 // [cap] unified row key of every lookup
    uint32_t* sort_id = nullptr;             // [cap] id of every lookup, for the bucket sorts
    uint2* rows = nullptr;                   // [cap] (row key, position) sorted by row
    float* partial = nullptr;    // [2 * chunks * CAFE_MAX_DIM] partial row sums of chunk-spanning rows
    int32_t* row_winner = nullptr;   // [hotn] migration: highest position that claims a hot row in this call (-1 between calls)
    uint2* rows_tmp = nullptr;       // [cap] pairs between two passes of the row sort
    int32_t* sort_scratch = nullptr; // radix-sort histograms
    cudaStream_t late = nullptr;     // importance of fields whose gradients arrive behind a gate
    cudaEvent_t ev_late = nullptr;
    // arrays whose side work a head start has already started (null: none)
    const uint32_t* begun_gid = nullptr;
    const int32_t* begun_row = nullptr;
    int begun_total = 0, begun_mode = 0;
};

int cafe_embed_ws_init(CafeEmbedWorkspace* ws, int cap, int hotn);
void cafe_embed_ws_free(CafeEmbedWorkspace* ws);

CafeSketchView cafe_internal_view(void* h);
CafeEmbedWorkspace* cafe_internal_ws(void* h);
// use_presort: the last cafe_internal_presort was for exactly these ids (and they have not changed since)
int cafe_internal_insert(void* h, const uint32_t* gid, const float* imp, const int* seg_off, int nseg, int32_t* mask,
                         int32_t* post_row, int mode, bool use_presort, cudaStream_t stream);
// starts the bucket sorts for an insert of `gid` beside whatever the caller queues next on `stream`.  `ids` holds the same
// ids in memory that stays as it is until the sorts are done (also: a further sort to run with them, or null).  A null gid
// withdraws an earlier presort.
void cafe_internal_presort(void* h, const uint32_t* gid, const uint32_t* ids, int n, const CafeSortDesc* also, cudaStream_t stream);
// makes `stream` wait for sorts that a presort started: before their inputs are written again (they stay outstanding for
// the call that uses them), or to use them
int cafe_internal_sort_wait(void* h, cudaStream_t stream);
int cafe_internal_sort_join(void* h, cudaStream_t stream);
// counts of segments >= seg of the next cafe_internal_insert are valid once `ev` has fired (null: no gate)
void cafe_internal_set_gate(void* h, int seg, cudaEvent_t ev);
void cafe_internal_set_error(const char* msg);

// ---- per-kernel timing and launch counting (prof.cu) ------------------------------------------------
enum {
    CAFE_P_FORWARD = 0, CAFE_P_NORM, CAFE_P_FIELDSUM, CAFE_P_IMPORTANCE, CAFE_P_LOOKUP_SORT, CAFE_P_MAIN, CAFE_P_SCAN,
    CAFE_P_LRU, CAFE_P_RESOLVE, CAFE_P_COMMIT, CAFE_P_REFIT, CAFE_P_MIGRATE, CAFE_P_ROWKEYS, CAFE_P_ROWSORT,
    CAFE_P_SCATTER, CAFE_P_FIXUP, CAFE_P_SEQ, CAFE_P_QUERY, CAFE_P_MEMSET, CAFE_P_OTHER, CAFE_P_MAIN_LATER, CAFE_P_MAIN_FINAL,
    CAFE_P_LRU_LATER, CAFE_P_PUSH, CAFE_P_IDS, CAFE_PROF_SLOTS
};
bool cafe_prof_serialise();
void cafe_prof_begin(int slot, cudaStream_t st);
void cafe_prof_end(cudaStream_t st);
struct CafeProfScope {
    cudaStream_t st;
    CafeProfScope(int slot, cudaStream_t s) : st(s) { cafe_prof_begin(slot, s); }
    ~CafeProfScope() { cafe_prof_end(st); }
};
#define CAFE_PROF(slot, stream) CafeProfScope cafe_prof_scope_##slot(slot, stream)
#define CAFE_PROF_DYN(slot, stream) CafeProfScope cafe_prof_scope_dyn(slot, stream)
