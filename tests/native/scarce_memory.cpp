// Calls that use more temporaries than they need, with one of them refused after
// another: what can do without must give the same result, and the rest must throw
// and leave the context usable. Run on a GPU, linked with the library's objects;
// exit status = number of failed checks.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <functional>
#include <memory>
#include <vector>

#include "runtime.hpp"
#include "segmented.hpp"

namespace gbc {
std::size_t static_map_insert(device_context& ctx, void* slots, std::size_t capacity, uint32_t empty_key, uint32_t empty_value,
                              const uint32_t* keys, const uint32_t* values, std::size_t n, std::size_t& not_placed);
void static_map_clear(device_context& ctx, void* slots, std::size_t capacity, uint32_t empty_key, uint32_t empty_value);
}  // namespace gbc

static int failures = 0;
#define CHECK(c)                                                                          \
    do {                                                                                  \
        if (!(c)) {                                                                       \
            ++failures;                                                                   \
            std::fprintf(stderr, "FAILED: %s at line %d (%s)\n", #c, __LINE__, g_what);   \
        }                                                                                 \
    } while (0)
static const char* g_what = "";

// Passes allocations on, but refuses number `refuse` (of those since reset).
struct scarce : gbc::memory_resource {
    std::shared_ptr<gbc::memory_resource> up;
    int refuse = -1, count = 0;
    bool as_unsupported = false;
    void* do_allocate(std::size_t b) override
    {
        if (count++ == refuse) {
            if (as_unsupported) throw gbc::unsupported_error("refused");
            throw gbc::out_of_memory("refused");
        }
        return up->allocate(b);
    }
    void do_deallocate(void* p, std::size_t b) noexcept override { up->deallocate(p, b); }
};

template <typename T> struct device_array {
    T* p = nullptr;
    std::size_t n;
    explicit device_array(std::size_t n_) : n(n_)
    {
        if (cudaMalloc(&p, n * sizeof(T)) != cudaSuccess) std::abort();
    }
    ~device_array() { cudaFree(p); }
    void put(const std::vector<T>& h) { cudaMemcpy(p, h.data(), n * sizeof(T), cudaMemcpyHostToDevice); }
    void clear() { cudaMemset(p, 0xEE, n * sizeof(T)); }
    std::vector<T> get() const
    {
        std::vector<T> h(n);
        cudaMemcpy(h.data(), p, n * sizeof(T), cudaMemcpyDeviceToHost);
        return h;
    }
};

static uint64_t mix(uint64_t x)
{
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

// Runs `call` with every allocation refused in turn, both ways; `same` compares
// what it left with what the undisturbed call did. Returns how many refusals
// the call did not survive.
static int refuse_each(gbc::device_context& ctx, scarce& mem, const char* what, const std::function<void()>& call,
                       const std::function<bool()>& same, bool unsupported_too)
{
    g_what = what;
    mem.refuse = -1;
    mem.count = 0;
    call();
    ctx.finish();
    const int total = mem.count;
    int thrown[2] = {};
    for (int way = 0; way < (unsupported_too ? 2 : 1); ++way)
        for (int k = 0; k < total; ++k) {
            mem.as_unsupported = way == 1;
            mem.refuse = k;
            mem.count = 0;
            bool threw = false;
            try {
                call();
            } catch (const gbc::out_of_memory&) {
                threw = true;
            } catch (const gbc::unsupported_error&) {
                threw = true;
            }
            ctx.finish();
            if (threw) ++thrown[way];
            else CHECK(same());
        }
    mem.refuse = -1;
    if (unsupported_too) CHECK(thrown[0] == thrown[1]);
    std::printf("%s: %d allocations, %d of them needed\n", what, total, thrown[0]);
    return thrown[0];
}

int main()
{
    auto config = gbc::default_arena_config(std::size_t(8) << 30);
    gbc::device_context ctx(0, nullptr, config, "");
    auto mem = std::make_shared<scarce>();
    mem->up = ctx.resource;
    ctx.resource = mem;

    // 64-bit sorts: below the size of the leading-digit form every temporary is
    // needed, above no more than those
    int needed = -1;
    for (std::size_t n : {(std::size_t(1) << 23) - 5, (std::size_t(1) << 23) + 5, (std::size_t(1) << 27) + 5}) {
        std::vector<uint64_t> keys(n);
        std::vector<uint32_t> vals(n);
        for (std::size_t i = 0; i < n; ++i) {
            keys[i] = mix(i);
            if (i % 1001 < 2) keys[i] = (keys[i] & 0xFFFFFFFFull) | (uint64_t(i / 100000000 + 1) << 33);  // long runs
            if (i % 777 == 0) keys[i] = 42;  // equal keys
            vals[i] = (uint32_t)i;
        }
        device_array<uint64_t> kin(n), kout(n);
        device_array<uint32_t> vin(n), vout(n);
        kin.put(keys);
        vin.put(vals);
        auto call = [&] { gbc::radix_sort(ctx, kin.p, kout.p, 8, 0, vin.p, vout.p, n, false); };
        call();
        ctx.finish();
        const std::vector<uint64_t> ek = kout.get();
        const std::vector<uint32_t> ev = vout.get();
        bool right = true;
        for (std::size_t i = 0; i < n; ++i) {
            right = right && keys[ev[i]] == ek[i];
            if (i > 0) right = right && (ek[i - 1] < ek[i] || (ek[i - 1] == ek[i] && ev[i - 1] < ev[i]));
        }
        g_what = "sort";
        CHECK(right);
        auto again = [&] {
            kout.clear();
            vout.clear();
            call();
        };
        auto same = [&] {
            const auto k = kout.get();
            const auto v = vout.get();
            return std::memcmp(k.data(), ek.data(), n * 8) == 0 && std::memcmp(v.data(), ev.data(), n * 4) == 0;
        };
        const int thrown = refuse_each(ctx, *mem, "sort", again, same, true);
        if (needed < 0) needed = thrown;
        CHECK(needed > 0 && thrown == needed);
    }
    {  // an insert by regions falls back to direct inserts
        const std::size_t cap = std::size_t(1) << 25, n = cap / 4;
        std::vector<uint32_t> keys(n);
        for (std::size_t i = 0; i < n; ++i) keys[i] = (uint32_t)i * 2654435761u;
        device_array<uint32_t> k(n);
        device_array<uint64_t> slots(cap);
        k.put(keys);
        std::size_t added = 0, left = 0;
        auto call = [&] {
            gbc::static_map_clear(ctx, slots.p, cap, 0xFFFFFFFFu, 0xFFFFFFFFu);
            added = gbc::static_map_insert(ctx, slots.p, cap, 0xFFFFFFFFu, 0xFFFFFFFFu, k.p, k.p, n, left);
        };
        CHECK(refuse_each(ctx, *mem, "static_map insert", call, [&] { return added == n && left == 0; }, false) == 0);
    }
    {  // the segmented scan's head bits
        const std::size_t n = (std::size_t(1) << 25) + 3;
        std::vector<int32_t> x(n);
        for (std::size_t i = 0; i < n; ++i) x[i] = (int32_t)(mix(i) % 7) - 3;
        const std::vector<uint32_t> off{0u, 10u, 20000000u, (uint32_t)n};
        device_array<int32_t> in(n), out(n);
        device_array<uint32_t> o(off.size());
        in.put(x);
        o.put(off);
        const int32_t zero = 0;
        std::vector<int32_t> expected(n);
        for (std::size_t s = 0; s + 1 < off.size(); ++s) {
            int32_t run = 0;
            for (std::size_t i = off[s]; i < off[s + 1]; ++i) expected[i] = run += x[i];
        }
        auto call = [&] {
            out.clear();
            gbc::segmented_scan(ctx, in.p, out.p, n, gbc::elem::i32, gbc::op_kind::plus, &zero, false, o.p, off.size() - 1);
        };
        CHECK(refuse_each(ctx, *mem, "segmented scan", call, [&] { return out.get() == expected; }, true) == 0);
    }
    ctx.resource = mem->up;
    return failures;
}
