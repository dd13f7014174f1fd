// dmap.cu -- DynamicMap<K,T>: a growing list of StaticMap submaps
// (include/dynamic_map.h, detail/dynamic_map/kernels.h).
//
// Same orchestration as the reference: inserts go to the active (last)
// submap; a new submap is added when the active one runs out of room (max
// load 0.6, minimum 10,000 spare, x2 growth), and may be prepared (cleared)
// ahead of time on a side stream; lookups fan out over the non-empty submaps
// and merge on the device; inserts into a grown map skip keys already present
// in an older submap (exact dedup) unless the caller promises unique keys.
#include <cmath>
#include <memory>
#include <new>
#include <vector>

#include "b2co_host.h"

using namespace b2co;

int b2co_oa_create_ex(b2co_oa_desc const* d, uint64_t requested, bool clear, b2co_stream stream, b2co_oa_table** out);
int b2co_oa_insert_counted(b2co_oa_table* t, void const* pairs, uint8_t const* stencil, uint64_t n, bool assign,
                           cudaStream_t s, uint64_t* counts);
int b2co_oa_mark(b2co_oa_table* t, void const* pairs, uint64_t n, bool assign, uint8_t* absent, cudaStream_t s);
int b2co_oa_lookup_over(b2co_oa_table* t, bool contains, void const* keys, void* out, uint64_t n, bool skip,
                        cudaStream_t s);

namespace {

cudaStream_t cs(b2co_stream s) { return reinterpret_cast<cudaStream_t>(s); }
b2co_stream bs(cudaStream_t s) { return reinterpret_cast<b2co_stream>(s); }

struct TableDel {
    void operator()(b2co_oa_table* t) const { b2co_oa_destroy(t); }
};
using TablePtr = std::unique_ptr<b2co_oa_table, TableDel>;

}  // namespace

struct b2co_dmap {
    static constexpr uint64_t kMinInsert = 10000;
    static constexpr double kMaxLoad = 0.60f;  // the reference stores it as a float
    static constexpr uint64_t kGrowth = 2;
    static constexpr uint64_t kSubBatch = 800000;

    b2co_oa_desc desc{};
    std::vector<TablePtr> submaps;
    std::vector<uint64_t> sizes;
    uint64_t size = 0, total_capacity = 0, next_capacity = 0;
    bool repeats = false;       // a key may be in two submaps: kAppendUnique took the caller's word, or +0 and -0
    uint8_t* absent = nullptr;  // one flag per pair of a batch: not in an older submap; grown on demand
    uint64_t absent_cap = 0;
    // background preparation of the next submap
    TablePtr next;
    uint64_t next_cap = 0;
    cudaStream_t prep = nullptr;
    cudaEvent_t prep_ev = nullptr;

    ~b2co_dmap()
    {
        if (next && prep) cudaStreamSynchronize(prep);
        next.reset();
        submaps.clear();
        if (absent) cudaFree(absent);
        if (prep_ev) cudaEventDestroy(prep_ev);
        if (prep) cudaStreamDestroy(prep);
    }

    uint32_t pair_bytes() const
    {
        uint32_t const raw = desc.key_bytes + desc.value_bytes;
        return raw <= 4 ? 4 : (raw <= 8 ? 8 : 16);
    }
    uint64_t capacity_of(size_t i) const
    {
        uint64_t c = 0;
        b2co_oa_capacity(submaps[i].get(), &c);
        return c;
    }
    uint64_t usable(uint64_t cap) const
    {
        uint64_t u = uint64_t(std::floor(double(float(kMaxLoad)) * double(cap)));
        return u > kMinInsert ? u - kMinInsert : 0;
    }
    size_t active() const { return submaps.size() - 1; }
    uint64_t active_room() const
    {
        uint64_t u = usable(capacity_of(active()));
        return u > sizes[active()] ? u - sizes[active()] : 0;
    }
    bool nonempty_before(size_t a) const
    {
        for (size_t s = 0; s < a; ++s)
            if (sizes[s]) return true;
        return false;
    }
    uint64_t grow_target(uint64_t min_usable) const
    {
        uint64_t g = size * kGrowth;
        return g > min_usable ? g : min_usable;
    }

    int add_submap(uint64_t requested, bool clear, cudaStream_t s, TablePtr& out)
    {
        b2co_oa_table* t = nullptr;
        if (int st = b2co_oa_create_ex(&desc, requested, clear, bs(s), &t)) return st;
        out.reset(t);
        return B2CO_OK;
    }

    int push(TablePtr t)
    {
        submaps.push_back(std::move(t));
        sizes.push_back(0);
        total_capacity += capacity_of(active());
        return B2CO_OK;
    }

    int discard_prepared()
    {
        if (next) {
            B2CO_CUDA(cudaStreamSynchronize(prep));
            next.reset();
        }
        next_cap = 0;
        return B2CO_OK;
    }

    // StartPrepareNext (dynamic_map.h:463-482): create the next submap and clear it on the side stream.
    int start_prepare(uint64_t min_usable)
    {
        if (next || !prep) return B2CO_OK;
        uint64_t cap = next_capacity;
        while (usable(cap) < grow_target(min_usable)) cap *= kGrowth;
        if (int st = add_submap(cap, false, prep, next)) return st;
        if (int st = b2co_oa_clear_async(next.get(), bs(prep))) return st;
        cudaError_t e = cudaEventRecord(prep_ev, prep);
        if (e != cudaSuccess) {
            discard_prepared();
            return cuda_fail(e, "DynamicMap::StartPrepareNext::cudaEventRecord");
        }
        next_cap = cap;
        return B2CO_OK;
    }

    // ActivateNext (dynamic_map.h:485-507).
    int activate_next(uint64_t min_usable, cudaStream_t s)
    {
        if (next && usable(next_cap) >= min_usable) {
            B2CO_CUDA(cudaStreamWaitEvent(s, prep_ev, 0));
            push(std::move(next));
            next_capacity = next_cap * kGrowth;
            next_cap = 0;
            return B2CO_OK;
        }
        if (int st = discard_prepared()) return st;
        uint64_t cap = next_capacity;
        while (usable(cap) < min_usable) cap *= kGrowth;
        TablePtr t;
        if (int st = add_submap(cap, true, s, t)) return st;
        push(std::move(t));
        next_capacity = cap * kGrowth;
        return B2CO_OK;
    }

    int ensure_active_room(uint64_t n, cudaStream_t s)
    {
        if (active_room() >= n) return B2CO_OK;
        return activate_next(grow_target(n), s);
    }

    // Flags the pairs whose key no older non-empty submap holds (BuildContainsMask,
    // dynamic_map.h:414-432, inverted); with `assign`, the older submaps that hold
    // a key take its new payload in the same pass.
    int build_absent(void const* pairs, uint64_t n, bool assign, cudaStream_t s)
    {
        if (absent_cap < n) {
            if (absent) cudaFree(absent);
            absent = nullptr;
            absent_cap = 0;
            B2CO_CUDA(cudaMalloc(&absent, n));
            absent_cap = n;
        }
        B2CO_CUDA(cudaMemsetAsync(absent, 1, n, s));
        for (size_t i = 0; i < active(); ++i) {
            if (!sizes[i]) continue;
            if (int st = b2co_oa_mark(submaps[i].get(), pairs, n, assign, absent, s)) return st;
        }
        return B2CO_OK;
    }

    // InsertChunk (dynamic_map.h:523-545).
    int insert_chunk(void const* pairs, uint64_t n, cudaStream_t s, uint64_t* inserted)
    {
        size_t a = active();
        uint64_t ins = 0;
        if (!nonempty_before(a)) {
            uint64_t failed = 0;
            if (int st = b2co_oa_insert(submaps[a].get(), pairs, n, bs(s), &failed)) return st;
            ins = n - failed;
        } else {
            uint64_t counts[3];  // failed, assigned, selected
            if (int st = build_absent(pairs, n, false, s)) return st;
            if (int st = b2co_oa_insert_counted(submaps[a].get(), pairs, absent, n, false, s, counts)) return st;
            ins = counts[2] - counts[0];
        }
        sizes[a] += ins;
        size += ins;
        *inserted = ins;
        return B2CO_OK;
    }

    // InsertOrAssignChunk (dynamic_map.h:549-575): only new keys are counted.
    int insert_or_assign_chunk(void const* pairs, uint64_t n, cudaStream_t s, uint64_t* inserted)
    {
        size_t a = active();
        uint64_t ins = 0;
        if (!nonempty_before(a)) {
            uint64_t failed = 0, assigned = 0;
            if (int st = b2co_oa_insert_or_assign(submaps[a].get(), pairs, n, bs(s), &failed, &assigned)) return st;
            ins = n - failed - assigned;
        } else {
            uint64_t counts[3];  // failed, assigned, selected
            if (int st = build_absent(pairs, n, true, s)) return st;
            if (int st = b2co_oa_insert_counted(submaps[a].get(), pairs, absent, n, true, s, counts)) return st;
            ins = counts[2] - counts[0] - counts[1];
        }
        sizes[a] += ins;
        size += ins;
        *inserted = ins;
        return B2CO_OK;
    }
};

int b2co_dmap_check(b2co_dmap const* m)
{
    if (!m || m->submaps.empty()) return fail(B2CO_ELOGIC, "DynamicMap is null or moved-from");
    return B2CO_OK;
}

// Find and Contains ask the newest non-empty submap first, which writes every
// output, and then the older ones, which write what they find: the answer of the
// oldest submap that has one stands, as when their answers are merged from the
// oldest on (kernels.h:73-112), without the merging passes and their buffer
// (Find of 16.8 M keys over three submaps: two passes of 75 us each).  A key that
// has been found is not asked for again where no other submap can hold it, which
// is so unless the caller's word was taken for it.
static int dmap_lookup(b2co_dmap* m, bool contains, void const* keys, void* out, uint64_t n, b2co_stream stream)
{
    if (int st = b2co_dmap_check(m)) return st;
    if (n == 0 || !keys || !out) return B2CO_OK;
    bool first = true;
    for (size_t i = m->submaps.size(); i-- > 0;) {
        if (!m->sizes[i] && !(i == 0 && first)) continue;  // an empty map asks its first submap
        b2co_oa_table* const t = m->submaps[i].get();
        int st = !first     ? b2co_oa_lookup_over(t, contains, keys, out, n, contains || !m->repeats, cs(stream))
                 : contains ? b2co_oa_contains_async(t, keys, static_cast<uint8_t*>(out), n, stream)
                            : b2co_oa_find_async(t, keys, out, n, stream);
        if (st) return st;
        first = false;
    }
    B2CO_CUDA(cudaStreamSynchronize(cs(stream)));
    return B2CO_OK;
}

extern "C" {

int b2co_dmap_create(b2co_oa_desc const* d, uint64_t initial_capacity, b2co_stream stream, b2co_dmap** out)
{
    if (!d || !out) return fail(B2CO_EINVAL, "null descriptor or output");
    *out = nullptr;
    if (d->value_bytes == 0) return fail(B2CO_EINVAL, "DynamicMap needs a payload (value_bytes > 0)");
    // the submaps check the layout and the key kind (2-byte keys with 2-byte
    // payloads; 4- and 8-byte keys with 4- or 8-byte payloads; integer or float)
    uint64_t kmask = d->key_bytes >= 8 ? ~0ull : ((1ull << (8 * d->key_bytes)) - 1);
    if ((d->empty_key_bits & kmask) == (d->erased_key_bits & kmask))
        return fail(B2CO_EINVAL, "DynamicMap: emptyKey and erasedKey must differ");
    auto* m = new (std::nothrow) b2co_dmap;
    if (!m) return fail(B2CO_ENOMEM, "host allocation failed");
    std::unique_ptr<b2co_dmap> guard(m);
    m->desc = *d;
    TablePtr t;
    if (int st = m->add_submap(initial_capacity, true, cs(stream), t)) return st;
    m->push(std::move(t));
    m->next_capacity = m->capacity_of(0) * b2co_dmap::kGrowth;
    m->repeats = d->key_kind != B2CO_KEY_INTEGER;
    // a failed side stream is not fatal: growth then happens synchronously
    if (cudaStreamCreateWithFlags(&m->prep, cudaStreamNonBlocking) == cudaSuccess) {
        if (cudaEventCreateWithFlags(&m->prep_ev, cudaEventDisableTiming) != cudaSuccess) {
            cudaStreamDestroy(m->prep);
            m->prep = nullptr;
        }
    } else {
        m->prep = nullptr;
    }
    *out = guard.release();
    return B2CO_OK;
}

int b2co_dmap_destroy(b2co_dmap* m)
{
    delete m;
    return B2CO_OK;
}

int b2co_dmap_size(b2co_dmap const* m, uint64_t* v)
{
    if (int st = b2co_dmap_check(m)) return st;
    *v = m->size;
    return B2CO_OK;
}

int b2co_dmap_capacity(b2co_dmap const* m, uint64_t* v)
{
    if (int st = b2co_dmap_check(m)) return st;
    *v = m->total_capacity;
    return B2CO_OK;
}

int b2co_dmap_num_submaps(b2co_dmap const* m, uint64_t* v)
{
    if (int st = b2co_dmap_check(m)) return st;
    *v = m->submaps.size();
    return B2CO_OK;
}

// Reserve (dynamic_map.h:142-166).
int b2co_dmap_reserve(b2co_dmap* m, uint64_t n, b2co_stream s)
{
    if (int st = b2co_dmap_check(m)) return st;
    uint64_t remaining = n;
    size_t idx = 0;
    while (remaining > 0) {
        uint64_t cap;
        if (idx < m->submaps.size()) {
            cap = m->capacity_of(idx);
        } else {
            cap = m->next_capacity;
            TablePtr t;
            if (int st = m->add_submap(cap, true, cs(s), t)) return st;
            m->push(std::move(t));
            m->next_capacity = cap * b2co_dmap::kGrowth;
        }
        uint64_t u = m->usable(cap);
        if (u >= remaining) break;
        remaining -= u;
        ++idx;
    }
    return B2CO_OK;
}

// Insert (dynamic_map.h:168-219).
int b2co_dmap_insert(b2co_dmap* m, void const* pairs, uint64_t n, int mode, b2co_stream stream, uint64_t* inserted)
{
    uint64_t dummy;
    if (!inserted) inserted = &dummy;
    *inserted = 0;
    if (int st = b2co_dmap_check(m)) return st;
    if (n == 0 || !pairs) return B2CO_OK;
    cudaStream_t s = cs(stream);
    if (int st = m->ensure_active_room(n, s)) return st;
    size_t a = m->active();
    uint32_t const pb = m->pair_bytes();
    if (mode == 1) {  // kAppendUnique: optimistic count, no per-batch sync
        m->repeats = true;
        for (uint64_t off = 0; off < n; off += b2co_dmap::kSubBatch) {
            uint64_t cur = n - off < b2co_dmap::kSubBatch ? n - off : b2co_dmap::kSubBatch;
            if (int st = b2co_oa_insert_async(m->submaps[a].get(), static_cast<char const*>(pairs) + off * pb, cur,
                                              stream))
                return st;
        }
        m->sizes[a] += n;
        m->size += n;
        *inserted = n;
        return B2CO_OK;
    }
    if (mode != 0) return fail(B2CO_EINVAL, "unknown DynamicMap insert mode");
    if (!m->nonempty_before(a)) {
        uint64_t failed = 0;
        if (int st = b2co_oa_insert(m->submaps[a].get(), pairs, n, stream, &failed)) return st;
        uint64_t ins = n >= failed ? n - failed : 0;
        m->sizes[a] += ins;
        m->size += ins;
        *inserted = ins;
        return B2CO_OK;
    }
    uint64_t total = 0, off = 0;
    while (off < n) {
        uint64_t room = m->active_room();
        if (room == 0) {
            if (int st = m->activate_next(m->grow_target(n - off), s)) return st;
            continue;
        }
        if (room < (n - off) * 2)
            if (int st = m->start_prepare(n - off)) return st;
        uint64_t chunk = n - off < room ? n - off : room, ins = 0;
        if (int st = m->insert_chunk(static_cast<char const*>(pairs) + off * pb, chunk, s, &ins)) return st;
        total += ins;
        off += chunk;
    }
    *inserted = total;
    return B2CO_OK;
}

// InsertOrAssign (dynamic_map.h:237-260): returns the number of new keys.
int b2co_dmap_insert_or_assign(b2co_dmap* m, void const* pairs, uint64_t n, b2co_stream stream, uint64_t* done)
{
    uint64_t dummy;
    if (!done) done = &dummy;
    *done = 0;
    if (int st = b2co_dmap_check(m)) return st;
    if (n == 0 || !pairs) return B2CO_OK;
    cudaStream_t s = cs(stream);
    if (int st = m->ensure_active_room(n, s)) return st;
    uint32_t const pb = m->pair_bytes();
    uint64_t total = 0, off = 0;
    while (off < n) {
        uint64_t room = m->active_room();
        if (room == 0) {
            if (int st = m->activate_next(m->grow_target(n - off), s)) return st;
            continue;
        }
        if (room < (n - off) * 2)
            if (int st = m->start_prepare(n - off)) return st;
        uint64_t chunk = n - off < room ? n - off : room, ins = 0;
        if (int st = m->insert_or_assign_chunk(static_cast<char const*>(pairs) + off * pb, chunk, s, &ins)) return st;
        total += ins;
        off += chunk;
    }
    *done = total;
    return B2CO_OK;
}

// Find (dynamic_map.h:262-290).
int b2co_dmap_find(b2co_dmap* m, void const* keys, void* out, uint64_t n, b2co_stream stream)
{
    return dmap_lookup(m, false, keys, out, n, stream);
}

// Contains (dynamic_map.h:292-316).
int b2co_dmap_contains(b2co_dmap* m, void const* keys, uint8_t* out, uint64_t n, b2co_stream stream)
{
    return dmap_lookup(m, true, keys, out, n, stream);
}

// Erase (dynamic_map.h:318-335).
int b2co_dmap_erase(b2co_dmap* m, void const* keys, uint64_t n, b2co_stream stream, uint64_t* erased)
{
    uint64_t dummy;
    if (!erased) erased = &dummy;
    *erased = 0;
    if (int st = b2co_dmap_check(m)) return st;
    if (n == 0 || !keys) return B2CO_OK;
    uint64_t total = 0;
    for (size_t i = 0; i < m->submaps.size(); ++i) {
        if (!m->sizes[i]) continue;
        uint64_t failed = 0;
        if (int st = b2co_oa_erase(m->submaps[i].get(), keys, n, stream, &failed)) return st;
        uint64_t del = n - failed;
        m->sizes[i] -= m->sizes[i] >= del ? del : m->sizes[i];
        total += del;
    }
    m->size -= m->size >= total ? total : m->size;
    *erased = total;
    return B2CO_OK;
}

// Clear (dynamic_map.h:349-357).
int b2co_dmap_clear(b2co_dmap* m, b2co_stream stream)
{
    if (int st = b2co_dmap_check(m)) return st;
    if (int st = m->discard_prepared()) return st;
    for (auto& t : m->submaps)
        if (int st = b2co_oa_clear(t.get(), stream)) return st;
    for (auto& x : m->sizes) x = 0;
    m->size = 0;
    m->repeats = m->desc.key_kind != B2CO_KEY_INTEGER;
    return B2CO_OK;
}

}  // extern "C"
