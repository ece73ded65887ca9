// Drives the library's internals where the public calls cannot reach a state:
//   status   a control block that a repair gave up on, through finish_repair (no GPU)
//   lists    repairs that start from a list of the test's own: only the winners of
//            their conflicts, and a list that becomes short and grows again; as one
//            kernel and as separate ones
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

// A repair under the independent-set rule of `states` from the worklist `list`,
// as one kernel (as far as it goes) or pass by pass. Returns how often the one
// kernel left a sweep to the others.
static uint32_t repair_from(sgc_handle* h, const std::vector<uint32_t>& states, const std::vector<uint32_t>& list,
                            bool fused, std::vector<uint32_t>& st, std::vector<uint64_t>& bm, sgc::RepairCtl& rc) {
    CHECK(sgc_upload(h, SGC_DL_STATES, states.data(), 4ull * h->n) == SGC_OK);
    rc = {};
    rc.mode = sgc::SWEEP_INDEP;
    rc.max_sweeps = 64;
    rc.list = rc.it = rc.cont = 1;
    const uint32_t count = (uint32_t)list.size();
    CHECK(cudaMemcpy(h->sb.rc, &rc, sizeof(rc), cudaMemcpyHostToDevice) == cudaSuccess);
    CHECK(cudaMemcpy(h->sb.wl, list.data(), 4ull * count, cudaMemcpyHostToDevice) == cudaSuccess);
    CHECK(cudaMemcpy(h->sb.wl_count, &count, 4, cudaMemcpyHostToDevice) == cudaSuccess);
    uint32_t left = 0;
    for (uint32_t k = 0; k < 70; k++) {
        if (fused) sgc::launch_repair_fused(h->g, h->sb, nullptr, h->stream, nullptr);
        CHECK(cudaMemcpyAsync(&rc, h->sb.rc, sizeof(rc), cudaMemcpyDeviceToHost, h->stream) == cudaSuccess);
        CHECK(cudaStreamSynchronize(h->stream) == cudaSuccess && !rc.fault);
        if (!rc.cont) break;
        left++;
        sgc::launch_repair_sweep(h->g, h->sb, sgc::SWEEP_INDEP, h->num_sms, h->stream);
        sgc::launch_repair_step(h->g, h->sb, h->num_sms, h->stream, nullptr);
    }
    CHECK(cudaGetLastError() == cudaSuccess && !rc.cont && rc.done);
    st.resize(h->n);
    bm.resize(h->n);
    CHECK(sgc_download(h, SGC_DL_STATES, st.data(), 4ull * h->n) == SGC_OK);
    CHECK(sgc_download(h, SGC_DL_BITMAPS, bm.data(), 8ull * h->n) == SGC_OK);
    return left;
}
// Both ways from the same start; the result is proper and the same.
static uint32_t both_ways(sgc_handle* h, const std::vector<uint32_t>& states, const std::vector<uint32_t>& list) {
    std::vector<uint64_t> start(h->n), bm1, bm2;
    std::vector<uint32_t> st1, st2;
    sgc::RepairCtl rc1, rc2;
    CHECK(sgc_download(h, SGC_DL_BITMAPS, start.data(), 8ull * h->n) == SGC_OK);
    const uint32_t left = repair_from(h, states, list, true, st1, bm1, rc1);
    sgc_validation v;
    CHECK(sgc_validate(h, &v) == SGC_OK && v.violations == 0 && v.uncolored_with_edges == 0);
    CHECK(sgc_upload(h, SGC_DL_BITMAPS, start.data(), 8ull * h->n) == SGC_OK);
    repair_from(h, states, list, false, st2, bm2, rc2);
    CHECK(st1 == st2 && bm1 == bm2 && rc1.it == rc2.it && rc1.need == rc2.need && rc1.next == rc2.next);
    return left;
}
static void lists() {
    sgc_repair_report rep{};
    // The winner y of a conflict with its neighbor x is listed, x is not: the first
    // sweep marks x and finds nobody who has to move.
    for (uint32_t n : {50u, 60000u, 400003u}) {
        const Rows r = ring(n);
        sgc_handle* h = make(r);
        CHECK(sgc_publish(h, &rep) == SGC_OK);
        std::vector<uint32_t> good(n);
        CHECK(sgc_download(h, SGC_DL_STATES, good.data(), 4ull * n) == SGC_OK);
        for (uint32_t pairs : {1u, 4u, 700u, 5000u}) {
            if (10 * pairs > n) continue;
            std::vector<uint32_t> states = good, list;
            const uint32_t apart = n / pairs;
            for (uint32_t i = 0; i < pairs; i++) {
                const uint32_t x = i * apart + 3, y = x + 1;  // the same degree: the higher id wins
                states[x] = states[y];
                list.push_back(y);
            }
            for (int k = 0; k < 20; k++) CHECK(both_ways(h, states, list) == 0);
        }
        sgc_destroy(h);
    }
    // 20 winners push 2,000 vertices (few enough for the first blocks: ids 8 apart,
    // so that no word of marks counts as crowded), which push 12,000 (too many).
    std::vector<std::vector<uint32_t>> adj(16000);
    auto join = [&](uint32_t a, uint32_t b) {
        adj[a].push_back(b);
        adj[b].push_back(a);
    };
    auto other = [](uint32_t k) { return 8 * (k / 7) + 1 + k % 7; };  // the ids between
    for (uint32_t l = 0; l < 2000; l++) {
        join(other(l % 20), 8 * l);
        for (uint32_t m = 0; m < 6; m++) join(8 * l, other(20 + 6 * l + m));
    }
    const Rows r(adj);
    sgc_handle* h = make(r);
    CHECK(sgc_publish(h, &rep) == SGC_OK);
    std::vector<uint32_t> list;
    for (uint32_t w = 0; w < 20; w++) list.push_back(other(w));
    CHECK(both_ways(h, std::vector<uint32_t>(r.n, 1u | 1u << 16), list) == 1);
    sgc_destroy(h);
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
    else if (!std::strcmp(what, "lists")) lists();
    else if (!std::strcmp(what, "give_up")) give_up();
    else return 2;
    return 0;
}
