// Drives the library's internals where the public calls cannot reach a state:
//   status   a control block that a repair gave up on, through finish_repair (no GPU)
//   give_up  a barrier that gives up at once (its failure word is set before the
//            call), through publish, core coloring and a batch's ticks
// Exits 0 when everything was as it should be.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../include/streamgc_batch.h"
#include "../../streamgc_b200/csrc/sgc_internal.h"

#define CHECK(c)                                                                             \
    do {                                                                                     \
        if (!(c)) {                                                                          \
            std::fprintf(stderr, "line %d: %s (last error: %s)\n", __LINE__, #c, sgc_last_error()); \
            std::exit(1);                                                                    \
        }                                                                                    \
    } while (0)

struct Rows {  // a host CSR
    std::vector<uint64_t> ptr{0};
    std::vector<uint32_t> col, deg;
    uint32_t n = 0;
    explicit Rows(const std::vector<std::vector<uint32_t>>& adj) : n((uint32_t)adj.size()) {
        for (const auto& r : adj) {
            col.insert(col.end(), r.begin(), r.end());
            ptr.push_back(col.size());
            deg.push_back((uint32_t)r.size());
        }
    }
};
static Rows ring(uint32_t n) {
    std::vector<std::vector<uint32_t>> adj(n);
    for (uint32_t v = 0; v < n; v++) adj[v] = {v ? v - 1 : n - 1, v + 1 < n ? v + 1 : 0};
    return Rows(adj);
}
static sgc_handle* make(const Rows& r, uint32_t flags = SGC_OPT_EXACT_SELECT) {
    StreamGCConfig cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.num_vertices = r.n;
    cfg.num_edges = r.col.size();
    cfg.epoch_size = 1024;
    cfg.histogram_threshold = 64;
    sgc_options o;
    sgc_default_options(&o);
    o.flags = flags;
    sgc_handle* h = nullptr;
    CHECK(sgc_create_ex(&cfg, &o, r.ptr.data(), r.col.data(), r.deg.data(), &h) == SGC_OK);
    return h;
}
static void set_failed(sgc_handle* h) {
    const uint32_t one = 1;
    CHECK(cudaMemcpy(&h->sb.bar->failed, &one, 4, cudaMemcpyHostToDevice) == cudaSuccess);
}

static void status() {
    sgc::RepairCtl rc{};
    rc.done = 1;  // the repair before this one ended proper
    sgc_handle h;
    h.h_rc_out = &rc;
    sgc_repair_report rep{};
    CHECK(sgci::finish_repair(&h, &rep) == SGC_OK && rep.proper == 1);
    rc.fault = 1;
    rep = {};
    CHECK(sgci::finish_repair(&h, &rep) == SGC_EDEVICE && rep.proper == 0);
}

static void give_up() {
    const Rows r = ring(3001);
    sgc_handle* h = make(r);
    std::vector<uint16_t> before(r.n), after(r.n);
    sgc_repair_report rep{};
    uint32_t colored = 0;
    CHECK(sgc_publish(h, &rep) == SGC_OK && rep.proper == 1);
    CHECK(sgc_publish(h, &rep) == SGC_OK && rep.incremental == 1);
    CHECK(sgc_download(h, SGC_DL_SNAPSHOT, before.data(), 2ull * r.n) == SGC_OK);
    for (int k = 0; k < 2; k++) {
        set_failed(h);
        CHECK(sgc_publish(h, &rep) == SGC_EDEVICE);
        CHECK(sgc_download(h, SGC_DL_SNAPSHOT, after.data(), 2ull * r.n) == SGC_OK && before == after);
    }
    CHECK(sgc_publish(h, &rep) == SGC_OK && rep.proper == 1 && rep.incremental == 0);
    CHECK(sgc_publish(h, &rep) == SGC_OK && rep.proper == 1 && rep.incremental == 1);
    set_failed(h);
    CHECK(sgc_color_core(h, 1, &colored) == SGC_EDEVICE);
    CHECK(sgc_color_core(h, 1, &colored) == SGC_OK);
    CHECK(sgc_publish(h, &rep) == SGC_OK && rep.proper == 1 && rep.incremental == 0);
    sgc_destroy(h);

    // the publish that writes its snapshot before it waits: a half written behind a
    // repair that gave up is not published, and both halves are whole afterwards
    h = make(r, SGC_OPT_EXACT_SELECT | SGC_OPT_GRAPH_PUBLISH);
    CHECK(sgc_publish(h, &rep) == SGC_OK);
    for (uint32_t k = 0; k < 12; k++) {
        std::vector<EdgeUpdate> ups(200);
        for (uint32_t i = 0; i < ups.size(); i++) {
            std::memset(&ups[i], 0, sizeof(EdgeUpdate));
            ups[i].u = (k * 977 + i * 13) % r.n;
            ups[i].v = (k * 389 + i * 29 + 7) % r.n;
            ups[i].type = SGC_UPDATE_ADD;
        }
        CHECK(sgc_apply(h, ups.data(), (uint32_t)ups.size(), SGC_MODE_CONCURRENT) == SGC_OK);
        CHECK(sgc_download(h, SGC_DL_SNAPSHOT, before.data(), 2ull * r.n) == SGC_OK);
        if (k % 3 == 1) {
            set_failed(h);
            CHECK(sgc_publish(h, &rep) == SGC_EDEVICE);
            CHECK(sgc_download(h, SGC_DL_SNAPSHOT, after.data(), 2ull * r.n) == SGC_OK && before == after);
        } else {
            CHECK(sgc_publish(h, &rep) == SGC_OK && rep.proper == 1);
            CHECK(sgc_download(h, SGC_DL_COLORS, before.data(), 2ull * r.n) == SGC_OK);
            CHECK(sgc_download(h, SGC_DL_SNAPSHOT, after.data(), 2ull * r.n) == SGC_OK && before == after);
        }
    }
    sgc_destroy(h);

    for (uint32_t flags : {SGC_BATCH_CUDA_GRAPH, 0u}) {
        sgc_batch_graph gr[2];
        std::memset(gr, 0, sizeof(gr));
        for (auto& g : gr) {
            g.num_vertices = r.n;
            g.row_ptr = r.ptr.data();
            g.col_idx = r.col.data();
        }
        sgc_batch_options o;
        sgc_batch_default_options(&o);
        o.flags = flags;
        o.max_tick_updates = 4096;
        sgc_batch* b = nullptr;
        CHECK(sgc_batch_create(gr, 2, &o, &b) == SGC_OK);
        sgc_handle* inner = *reinterpret_cast<sgc_handle**>(b);  // the batch's first member
        sgc_batch_tick_report t{};
        sgc_batch_close_epochs(b);
        CHECK(sgc_batch_tick(b, &t) == SGC_OK && t.proper == 1 && t.published == 2);
        set_failed(inner);
        sgc_batch_close_epochs(b);
        CHECK(sgc_batch_tick(b, &t) == SGC_EDEVICE);
        CHECK(sgc_batch_publish_count(b, 0) == 1 && sgc_batch_publish_count(b, 1) == 1);
        CHECK(sgc_batch_tick(b, &t) == SGC_OK && t.proper == 1 && t.published == 2);  // the epochs close now
        CHECK(sgc_batch_publish_count(b, 0) == 2);
        sgc_batch_destroy(b);
    }
}

int main(int argc, char** argv) {
    const char* what = argc > 1 ? argv[1] : "";
    if (!std::strcmp(what, "status")) status();
    else if (!std::strcmp(what, "give_up")) give_up();
    else return 2;
    return 0;
}
