// Failure paths of the library's host code, on the stand-in runtime of
// fake_cudart.cpp: host_faults CASE exits 0 if the case holds.
#include <sys/mman.h>
#include <unistd.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <set>
#include <string>
#include <vector>

#include "aieplace.h"
#include "fake_cudart.h"

#define REQUIRE(cond)                                                         \
    do {                                                                      \
        if (!(cond)) {                                                        \
            fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #cond);        \
            exit(1);                                                          \
        }                                                                     \
    } while (0)

namespace {

// A netlist whose internal order (movable, fixed with area, fixed without) is not
// its own: every third node is fixed, every fourth of those without area.
struct Netlist {
    std::vector<int32_t> ptr{0}, pin;
    std::vector<float> w, h, x, y;
    std::vector<uint8_t> fixed;
    ap_netlist nl{};
    explicit Netlist(int n = 60, float die = 64.f) {
        for (int i = 0; i < n; ++i) {
            const bool f = i % 3 == 0;
            fixed.push_back(f);
            w.push_back(f && i % 12 == 0 ? 0.f : 1.f);
            h.push_back(1.f);
            x.push_back((float)(i % 8));
            y.push_back((float)(i / 8));
        }
        for (int i = 0; i + 1 < n; ++i) {
            pin.push_back(i);
            pin.push_back(i + 1);
            ptr.push_back((int32_t)pin.size());
        }
        nl.num_nodes = n;
        nl.num_nets = n - 1;
        nl.num_pins = (int32_t)pin.size();
        nl.net_ptr = ptr.data();
        nl.pin_node = pin.data();
        nl.node_w = w.data();
        nl.node_h = h.data();
        nl.node_x = x.data();
        nl.node_y = y.data();
        nl.node_fixed = fixed.data();
        nl.die_xh = nl.die_yh = die;
    }
    std::vector<int> order(int fillers) const {
        std::vector<int> o;
        for (int cls = 0; cls < 3; ++cls) {
            for (int i = 0; i < nl.num_nodes; ++i)
                if ((!fixed[i] ? 0 : w[i] * h[i] > 0.f ? 1 : 2) == cls) o.push_back(i);
            if (cls == 0) o.insert(o.end(), (size_t)fillers, -1);
        }
        return o;
    }
};

ap_params params(int bins, int solver = AP_FIELD_FP32) {
    ap_params p;
    ap_params_default(&p);
    p.bins_x = p.bins_y = bins;
    p.field_solver = solver;
    return p;
}

ap_handle *create(const Netlist &n, const ap_params &p) {
    ap_handle *h = nullptr;
    REQUIRE(ap_create(&n.nl, &p, &h) == AP_OK && h);
    return h;
}

// Calls on host arrays need no memory that ap_create did not take, and what they
// read on the device has arrived: whichever allocation fails, every call passes, and
// its kernels get the netlist's order.
void host_arrays() {
    fake::watch("import_kernel", 1);
    fake::watch("export_positions_kernel", 1);
    fake::watch("export_gradient_kernel", 1);
    fake::watch("export_force_kernel", 2);
    for (int fillers = 0; fillers < 2; ++fillers)
        for (int fail = 0; fail <= 3; ++fail) {
            const Netlist n;
            ap_params p = params(32);
            p.filler_cells = fillers;
            ap_handle *h = create(n, p);
            int32_t n_fill = 0;
            REQUIRE(ap_get_fillers(h, &n_fill, nullptr, nullptr) == AP_OK && (n_fill > 0) == (fillers > 0));
            const std::vector<int> order = n.order(n_fill);
            std::vector<float> x(n.x), y(n.y), gx(x.size()), gy(x.size()), field(32 * 32);
            double hp, wa;
            fake::fail_malloc(fail);
            fake::take_launches();
            for (int attempt = 0; attempt < 3; ++attempt) {
                REQUIRE(ap_init_positions(h, n.x.data(), n.y.data()) == AP_OK);
                REQUIRE(ap_get_positions(h, x.data(), y.data()) == AP_OK);
                REQUIRE(ap_wirelength_grad(h, n.x.data(), n.y.data(), 4.f, gx.data(), gy.data(), &hp, &wa) == AP_OK);
                REQUIRE(ap_node_force(h, n.x.data(), n.y.data(), field.data(), field.data(), 4.f, 1.f, gx.data(),
                                      gy.data(), nullptr, nullptr) == AP_OK);
            }
            int seen = 0;
            for (const fake::Launch &l : fake::take_launches())
                for (const void *q : l.ptr) {
                    REQUIRE(q && fake::is_device(q));
                    REQUIRE(!memcmp(q, order.data(), sizeof(int) * order.size()));
                    REQUIRE(!l.early);
                    ++seen;
                }
            REQUIRE(seen == 3 * 6);  // an import each but for the read-back, an export each but for the first
            fake::fail_malloc(0);
            REQUIRE(ap_destroy(h) == AP_OK);
        }
}

// ap_create takes everything or nothing.
void create_fails() {
    const Netlist n;
    ap_params p = params(32);
    p.filler_cells = 1;
    ap_destroy(create(n, p));
    const int before = fake::mallocs();
    ap_destroy(create(n, p));
    const int count = fake::mallocs() - before;
    const size_t held = fake::live_bytes();
    for (int k = 1; k <= count; ++k) {
        ap_handle *h = nullptr;
        fake::fail_malloc(k);
        REQUIRE(ap_create(&n.nl, &p, &h) == AP_ERR_CUDA && !h);
        REQUIRE(fake::live_bytes() == held);
        fake::fail_malloc(0);
        ap_create(&n.nl, &p, &h);  // may report what is left of the first error
        if (h) ap_destroy(h);
        ap_destroy(create(n, p));
    }
}

// The tensor-core solve is made whole or not at all: whichever allocation or copy
// fails, the call says so and keeps nothing, and the next one makes all of it.
void tensor_cores_retry() {
    const Netlist n;
    fake::watch("split_kernel", 1);
    fake::watch("split_kernel", 2);
    fake::watch("split_kernel", 3);
    const auto splits = [](int count) {
        int seen = 0;
        for (const fake::Launch &l : fake::take_launches())
            if (!l.ptr.empty()) {
                for (const void *q : l.ptr) REQUIRE(q && fake::is_device(q));
                ++seen;
            }
        REQUIRE(seen == count);
    };
    int allocations = 0;
    for (int what = 0; what < 2; ++what)
        for (int k = 1;; ++k) {
            ap_handle *h = create(n, params(128, AP_FIELD_BF16X3));
            const size_t held = fake::live_bytes();
            fake::take_launches();
            (what ? fake::fail_upload : [](int f) { fake::fail_malloc(f); })(k);
            const int before = fake::mallocs();
            const int r = ap_debug_inject(h, AP_FAULT_TC_STALL, 1000000);
            const bool failed = r != AP_OK;
            if (failed) {
                REQUIRE(r == AP_ERR_CUDA);
                REQUIRE(fake::live_bytes() == held);
                fake::take_launches();
                REQUIRE(ap_debug_inject(h, AP_FAULT_TC_STALL, 1000000) == AP_OK);
            } else if (what == 0) {
                allocations = fake::mallocs() - before;
            }
            splits(3);  // C, C^T and S^T
            std::vector<float> d(128 * 128, 1.f), ex(d), ey(d);
            fake::fail_malloc(0);
            fake::fail_upload(0);
            REQUIRE(ap_field_solve(h, d.data(), ex.data(), ey.data(), AP_FIELD_BF16X3) == AP_OK);
            REQUIRE(ap_destroy(h) == AP_OK);
            if (!failed) break;
        }
    REQUIRE(allocations >= 21);  // two input maps, 16 maps, three of the persistent solve
}

int launches_of(const char *kernel) {
    int seen = 0;
    for (const fake::Launch &l : fake::take_launches()) seen += l.name.find(kernel) != std::string::npos;
    return seen;
}

// ap_solver_info reports on an optional path: where that cannot be made it says so
// and the handle works on, and it never changes which solver the handle runs.
void solver_info() {
    const Netlist n;
    std::vector<float> d(128 * 128, 1.f), ex(d), ey(d);
    for (int solver : {AP_FIELD_FP32, AP_FIELD_BF16X3}) {
        ap_handle *h = create(n, params(128, solver));
        int32_t variant = 7, tile = 0;
        float tc_ms[5], simt_ms[2] = {0.f, 0.f};
        fake::fail_malloc(3, true);
        REQUIRE(ap_solver_info(h, &variant, tc_ms, &tile, simt_ms) == AP_OK);
        REQUIRE(variant == -1 && tile == 32 && simt_ms[0] > 0.f && simt_ms[1] == -1.f);
        fake::fail_malloc(0);
        REQUIRE(ap_field_solve(h, d.data(), ex.data(), ey.data(), solver) == AP_OK);
        setenv("AP_TC_VARIANT", "1", 1);  // too late for this handle
        REQUIRE(ap_solver_info(h, &variant, tc_ms, nullptr, nullptr) == AP_OK && variant >= 0 && tc_ms[1] > 0.f);
        unsetenv("AP_TC_VARIANT");
        fake::take_launches();
        REQUIRE(ap_field_solve(h, d.data(), ex.data(), ey.data(), solver) == AP_OK);
        REQUIRE(launches_of("split_kernel") == 0);
        REQUIRE(ap_destroy(h) == AP_OK);
    }
    setenv("AP_TC_VARIANT", "1", 1);
    ap_handle *h = create(n, params(128, AP_FIELD_BF16X3));
    unsetenv("AP_TC_VARIANT");
    int32_t variant = 7;
    REQUIRE(ap_solver_info(h, &variant, nullptr, nullptr, nullptr) == AP_OK && variant == 1);
    fake::take_launches();
    REQUIRE(ap_field_solve(h, d.data(), ex.data(), ey.data(), -1) == AP_OK);
    REQUIRE(launches_of("split_kernel") == 1);
    REQUIRE(ap_destroy(h) == AP_OK);
}

// An output that is no host memory is the runtime's to refuse: the host does not
// write to it.
void device_output() {
    const Netlist n;
    ap_handle *h = create(n, params(64));
    std::vector<float> d(64 * 64, 1.f), e(d);
    void *dev = fake::device_only(64 * 64 * 8);
    REQUIRE(ap_density_map(h, n.x.data(), n.y.data(), (int64_t *)dev) == AP_ERR_CUDA);
    REQUIRE(ap_field_solve(h, d.data(), (float *)dev, e.data(), -1) != AP_OK);
    ap_field_solve(h, d.data(), e.data(), e.data(), -1);  // may report what is left of the error
    REQUIRE(ap_field_solve(h, d.data(), e.data(), e.data(), -1) == AP_OK);
    REQUIRE(ap_destroy(h) == AP_OK);
    ap_surrogate_config c;
    ap_surrogate *s = nullptr;
    REQUIRE(ap_surrogate_config_default(&c) == AP_OK && ap_surrogate_create(&c, &s) == AP_OK);
    std::vector<float> x((c.factor * c.factor + 2) * 16 * 16);
    REQUIRE(ap_surrogate_forward(s, x.data(), 1, 16, (float *)dev) == AP_ERR_CUDA);
    REQUIRE(ap_surrogate_destroy(s) == AP_OK);
}

// What a kernel's shared memory is allowed holds for the whole process: a batch of
// small grids must not take back what a batch of large ones, in another thread, is
// about to launch with.
void shared_memory_limits() {
    const Netlist n;
    ap_batch *large = nullptr, *small = nullptr;
    const ap_params pl = params(4096), ps = params(64);
    REQUIRE(ap_create_batch(1, &n.nl, &pl, &large) == AP_OK);
    REQUIRE(ap_create_batch(1, &n.nl, &ps, &small) == AP_OK);
    const fake::SmemLimit s = fake::smem_limit("persist_field_kernelILi512E");
    REQUIRE(s.most > 0 && s.last == s.most);
    REQUIRE(ap_batch_destroy(small) == AP_OK && ap_batch_destroy(large) == AP_OK);
}

// The graph of four trials is made by the first call that can use it: where that
// fails the loop runs on the graph of one, which the initial placement made.
void trial_graphs() {
    const Netlist n;
    ap_handle *h = create(n, params(32));
    REQUIRE(ap_init_positions(h, n.x.data(), n.y.data()) == AP_OK);
    const auto launches = [&](int trials) {
        const int before = fake::graph_launches();
        REQUIRE(ap_step_async(h, trials) == AP_OK);
        return fake::graph_launches() - before;
    };
    fake::fail_instantiate(1, true);
    REQUIRE(launches(10) == 10);
    REQUIRE(launches(3) == 3);
    fake::fail_instantiate(0);
    REQUIRE(launches(10) == 2 + 2);
    REQUIRE(launches(3) == 3);
    REQUIRE(ap_init_positions(h, n.x.data(), n.y.data()) == AP_OK);
    REQUIRE(launches(8) == 2);
    REQUIRE(ap_destroy(h) == AP_OK);
}

// ap_profile_stages times the loop's own kernels.
void profile_launches() {
    const Netlist n;
    const auto names = [] {
        std::multiset<std::string> s;
        for (const fake::Launch &l : fake::take_launches()) s.insert(l.name);
        return s;
    };
    for (int c = 0; c < 5; ++c) {
        ap_params p = params(c == 0 ? 32 : c < 3 ? 64 : 128, c < 3 ? AP_FIELD_FP32 : AP_FIELD_BF16X3);
        p.filler_cells = c == 2;
        p.use_graph = 0;
        if (c == 4) setenv("AP_TC_VARIANT", "1", 1);
        ap_handle *h = create(n, p);
        unsetenv("AP_TC_VARIANT");
        REQUIRE(ap_init_positions(h, n.x.data(), n.y.data()) == AP_OK);
        names();
        REQUIRE(ap_step_async(h, 1) == AP_OK);
        const auto loop = names();
        float ms[8];
        int32_t stages = 0;
        REQUIRE(ap_profile_stages(h, 1, ms, &stages) == AP_OK && stages == 5);
        REQUIRE(!loop.empty() && names() == loop);
        REQUIRE((ms[1] > 0.f) == (c == 4) && ms[0] > 0.f && ms[2] > 0.f && ms[3] > 0.f && ms[4] > 0.f);
        REQUIRE(ap_destroy(h) == AP_OK);
    }
}

// What a call puts on the null stream has arrived before anything of the library's
// non-blocking streams is launched.
void null_stream_waits() {
    const Netlist n;
    const auto waited = [](const char *what) {
        if (fake::early_launches()) {
            fprintf(stderr, "%s: %d launches too early\n", what, fake::early_launches());
            exit(1);
        }
    };
    std::vector<float> d(128 * 128, 1.f), ex(d), ey(d);
    for (int pinned = 0; pinned < 2; ++pinned) {
        if (pinned) setenv("AP_TC_VARIANT", "1", 1);
        ap_handle *h = create(n, params(128, AP_FIELD_BF16X3));
        unsetenv("AP_TC_VARIANT");
        REQUIRE(ap_init_positions(h, n.x.data(), n.y.data()) == AP_OK && ap_step_async(h, 5) == AP_OK);
        waited("ap_create, ap_init_positions");
        size_t bytes = 0;
        REQUIRE(ap_snapshot_size(h, &bytes) == AP_OK);
        std::vector<char> blob(bytes);
        REQUIRE(ap_snapshot(h, blob.data(), bytes) == AP_OK && ap_restore(h, blob.data(), bytes) == AP_OK);
        REQUIRE(ap_step_async(h, 1) == AP_OK);
        waited("ap_restore");
        REQUIRE(ap_debug_inject(h, AP_FAULT_TC_STALL, 1000000) == AP_OK && ap_debug_inject(h, AP_FAULT_NONE, 0) == AP_OK);
        REQUIRE(ap_field_solve(h, d.data(), ex.data(), ey.data(), -1) == AP_OK);
        waited("ap_debug_inject");
        ap_surrogate_config c;
        ap_surrogate *s = nullptr;
        REQUIRE(ap_surrogate_config_default(&c) == AP_OK && ap_surrogate_create(&c, &s) == AP_OK);
        REQUIRE(ap_attach_surrogate(h, s, nullptr) == AP_OK && ap_step_async(h, 1) == AP_OK);
        waited("ap_surrogate_create, ap_attach_surrogate");
        int32_t np = 0;
        REQUIRE(ap_surrogate_num_params(s, &np) == AP_OK);
        std::vector<float> w((size_t)np);
        REQUIRE(ap_surrogate_set_params(s, w.data(), np) == AP_OK && ap_step_async(h, 1) == AP_OK);
        waited("ap_surrogate_set_params");
        REQUIRE(ap_destroy(h) == AP_OK && ap_surrogate_destroy(s) == AP_OK);
    }
    for (int solver : {AP_FIELD_FP32, AP_FIELD_BF16X3}) {
        const ap_params p[2] = {params(128, solver), params(128, solver)};
        const ap_netlist nl[2] = {n.nl, n.nl};
        ap_batch *b = nullptr;
        REQUIRE(ap_create_batch(2, nl, p, &b) == AP_OK);
        waited("ap_create_batch");
        REQUIRE(ap_batch_init_seeded(b, 1, 1.f) == AP_OK && ap_batch_step(b, 2) == AP_OK);
        waited("ap_batch_init_seeded");
        if (solver == AP_FIELD_FP32) {
            REQUIRE(ap_batch_set_item_blocks(b, 1) == AP_OK && ap_batch_step(b, 1) == AP_OK);
            waited("ap_batch_set_item_blocks");
            REQUIRE(ap_batch_debug_inject(b, AP_FAULT_NONE, 0) == AP_OK && ap_batch_step(b, 1) == AP_OK);
            waited("ap_batch_debug_inject");
        }
        REQUIRE(ap_batch_destroy(b) == AP_OK);
    }
}

// A batch of few work items launches no more blocks than it has items, and of the
// kernels that come in several occupancies the one without spilled registers.
void batch_blocks() {
    const Netlist n;
    const ap_params p[3] = {params(32), params(64), params(32)};
    const ap_netlist nl[3] = {n.nl, n.nl, n.nl};
    ap_batch *b = nullptr;
    REQUIRE(ap_create_batch(3, nl, p, &b) == AP_OK && ap_batch_init_seeded(b, 1, 1.f) == AP_OK);
    ap_batch_info info;
    float ms[6];
    REQUIRE(ap_batch_get_info(b, &info) == AP_OK && info.form == AP_BATCH_PERSISTENT);
    fake::take_launches();
    REQUIRE(ap_batch_profile(b, 1, ms) == AP_OK);
    const char *stage[6] = {"persist_update_kernelILi3E", "persist_scatter_kernel", "persist_rho_kernel", "persist_wa_kernel",
                            "persist_field_kernel", "persist_gather_kernelILi4E"};
    int seen = 0;
    for (const fake::Launch &l : fake::take_launches())
        for (int k = 0; k < 6; ++k)
            if (l.name.find(stage[k]) != std::string::npos) {
                REQUIRE(l.blocks >= 1 && (int)l.blocks <= info.items[k]);
                ++seen;
            }
    REQUIRE(seen == 6);
    REQUIRE(ap_batch_destroy(b) == AP_OK);
}

// Small designs: a call on host arrays waits for the device once, a network's
// inference not beyond its read-back.
void small_calls() {
    const Netlist n;
    ap_handle *h = create(n, params(32));
    std::vector<float> x(n.x), y(n.y), gx(x), gy(x), field(32 * 32);
    std::vector<int64_t> rho(32 * 32);
    double hp, wa;
    REQUIRE(ap_init_positions(h, x.data(), y.data()) == AP_OK);
    const auto waits = [](const std::function<int()> &call) {
        const int before = fake::stream_waits();
        REQUIRE(call() == AP_OK);
        return fake::stream_waits() - before;
    };
    REQUIRE(waits([&] { return ap_get_positions(h, x.data(), y.data()); }) == 1);
    REQUIRE(waits([&] { return ap_density_map(h, x.data(), y.data(), rho.data()); }) == 1);
    REQUIRE(waits([&] {
                return ap_wirelength_grad(h, x.data(), y.data(), 4.f, gx.data(), gy.data(), &wa, &hp);
            }) == 1);
    REQUIRE(waits([&] {
                return ap_node_force(h, x.data(), y.data(), field.data(), field.data(), 4.f, 1.f, gx.data(), gy.data(),
                                     nullptr, nullptr);
            }) == 1);
    REQUIRE(ap_destroy(h) == AP_OK);
    ap_surrogate_config c;
    ap_surrogate *s = nullptr;
    REQUIRE(ap_surrogate_config_default(&c) == AP_OK && ap_surrogate_create(&c, &s) == AP_OK);
    std::vector<float> in((c.factor * c.factor + 2) * 16 * 16), out(2 * c.factor * c.factor * 16 * 16);
    REQUIRE(waits([&] { return ap_surrogate_forward(s, in.data(), 1, 16, out.data()); }) == 0);
    REQUIRE(ap_surrogate_destroy(s) == AP_OK);
}

// Results end where the caller's memory does: between pages that fault, at every
// offset of the end, and past the size from which pages are no longer touched first.
void outputs_in_bounds() {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    const Netlist n;
    for (int bins : {32, 64}) {
        ap_handle *h = create(n, params(bins));
        const size_t bytes = sizeof(int64_t) * bins * bins, span = (bytes + page - 1) / page * page;
        char *m = (char *)mmap(nullptr, span + 2 * page, PROT_NONE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
        REQUIRE(m != MAP_FAILED && mprotect(m + page, span, PROT_READ | PROT_WRITE) == 0);
        memset(m + page, 7, span);
        REQUIRE(ap_density_map(h, n.x.data(), n.y.data(), (int64_t *)(m + page + span - bytes)) == AP_OK);
        for (size_t i = 0; i < span - bytes; ++i) REQUIRE(m[page + i] == 7);
        REQUIRE(ap_density_map(h, n.x.data(), n.y.data(), (int64_t *)(m + page)) == AP_OK);
        munmap(m, span + 2 * page);
        REQUIRE(ap_destroy(h) == AP_OK);
    }
    ap_surrogate_config c;
    ap_surrogate *s = nullptr;
    REQUIRE(ap_surrogate_config_default(&c) == AP_OK);
    c.factor = 1;
    REQUIRE(ap_surrogate_create(&c, &s) == AP_OK);
    for (int res : {16, 48, 512}) {
        for (int batch : {1, 3, 24, 25}) {  // 24 and 25 maps of 512: 48 MB and beyond
            const size_t px = (size_t)batch * res * res, bytes = sizeof(float) * 2 * px, span = (bytes + page - 1) / page * page;
            std::vector<float> in(3 * px);
            char *m = (char *)mmap(nullptr, span + 2 * page, PROT_NONE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
            REQUIRE(m != MAP_FAILED && mprotect(m + page, span, PROT_READ | PROT_WRITE) == 0);
            REQUIRE(ap_surrogate_forward(s, in.data(), batch, res, (float *)(m + page + span - bytes)) == AP_OK);
            munmap(m, span + 2 * page);
        }
    }
    REQUIRE(ap_surrogate_destroy(s) == AP_OK);
}

const std::map<std::string, std::function<void()>> kCases = {
    {"host_arrays", host_arrays},
    {"create_fails", create_fails},
    {"tensor_cores_retry", tensor_cores_retry},
    {"solver_info", solver_info},
    {"device_output", device_output},
    {"shared_memory_limits", shared_memory_limits},
    {"trial_graphs", trial_graphs},
    {"profile_launches", profile_launches},
    {"null_stream_waits", null_stream_waits},
    {"batch_blocks", batch_blocks},
    {"small_calls", small_calls},
    {"outputs_in_bounds", outputs_in_bounds},
};

}  // namespace

int main(int argc, char **argv) {
    if (argc < 2 || !kCases.count(argv[1])) return 2;
    kCases.at(argv[1])();
    return 0;
}
