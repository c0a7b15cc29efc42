// The library's host code on a device of host memory (fake_device.h): host_paths <check>.
#include "fake_device.h"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <string>
#include <vector>

static int fails = 0;

static void check(bool ok, const std::string& what)
{
    if (!ok) std::printf("FAIL %s\n", what.c_str());
    fails += ok ? 0 : 1;
}

struct Made {
    std::vector<float> xyz, w;
    std::vector<int32_t> from, to;
    nc_params p{};
    int32_t n;
    explicit Made(int32_t neurons, int32_t synapses, int mode = NC_STEP_DENSE) : n(neurons)
    {
        nc_default_params(&p);
        p.step_mode = mode;
        for (int32_t i = 0; i < 3 * n; ++i) xyz.push_back((float)(i * 7919 % 101) / 40.0f);
        for (int32_t k = 0; k < synapses; ++k) {
            from.push_back(k * 31 % n);
            to.push_back(k * 17 % n);
            w.push_back((float)(k + 1) / (float)(synapses + 1));
        }
    }
    nc_net* create()
    {
        nc_net* net = nullptr;
        const int rc = nc_create(n, xyz.data(), (int64_t)w.size(), from.data(), to.data(), w.data(), nullptr, nullptr, &p, &net);
        check(rc == NC_OK, std::string("create: ") + nc_last_error());
        return net;
    }
    nc_net_spec spec(int32_t horizon)
    {
        nc_net_spec s{};
        s.n_neurons = n;
        s.xyz = xyz.data();
        s.n_synapses = (int64_t)w.size();
        s.syn_from = from.data();
        s.syn_to = to.data();
        s.syn_weight = w.data();
        s.params = p;
        s.horizon = horizon;
        return s;
    }
    // weights read back: as given, NaN where a pair is repeated
    bool same(const std::vector<float>& got) const
    {
        for (size_t k = 0; k < w.size(); ++k)
            if (!(got[k] == w[k] || std::isnan(got[k]))) return false;
        return true;
    }
};

// Weights read for the first time, however late the legacy stream's work is done.
static void weights_order()
{
    for (int delay : {0, 1, 2, 3, 5, 9, 1000}) {
        fake::legacy_delay = delay;
        Made m(50, 400);
        std::vector<float> got(m.w.size());
        nc_net* net = m.create();
        check(nc_read_weights(net, got.data()) == NC_OK && m.same(got), "weights, delay " + std::to_string(delay));
        nc_destroy(net);
        nc_net_spec specs[2] = {m.spec(5), m.spec(9)};
        nc_batch* b = nullptr;
        check(nc_batch_create(2, specs, &b) == NC_OK, "batch");
        for (int32_t q = 0; q < 2; ++q)
            check(nc_batch_read_weights(b, q, got.data()) == NC_OK && m.same(got), "batch weights, delay " + std::to_string(delay));
        nc_batch_destroy(b);
    }
    check(fake::faults == 0, "positions out of range");
}

// The raster's rows are cleared before the steps that write them.
static void raster_order()
{
    for (int delay = 0; delay < 24; ++delay) {
        fake::legacy_delay = delay;
        Made m(64, 300);
        nc_net* net = m.create();
        std::vector<uint8_t> rows(5 * 8, 0);
        int32_t steps = 0;
        check(nc_record_raster(net, 5) == NC_OK && nc_run(net, 4) == NC_OK, "run");
        check(nc_read_raster(net, rows.data(), (int64_t)rows.size(), &steps) == NC_OK && steps == 4, "read");
        check(rows == std::vector<uint8_t>([] { std::vector<uint8_t> v(32, 0xff); v.resize(40, 0); return v; }()),
              "rows of the steps, delay " + std::to_string(delay));
        nc_destroy(net);
    }
    check(fake::faults == 0, "rows out of range");
}

// A raster that cannot be replaced for want of memory is no longer written.
static void raster_refused()
{
    Made m(64, 300);
    nc_net* net = m.create();
    check(nc_record_raster(net, 5) == NC_OK && nc_run(net, 2) == NC_OK, "run");
    fake::fail_malloc_from = 8 * 70;
    check(nc_record_raster(net, 70) == NC_ERR_NOMEM, "refused");
    check(nc_run(net, 2) == NC_OK && fake::faults == 0, "steps after it");
    int32_t steps = -1;
    uint8_t none[1];
    check(nc_read_raster(net, none, 1, &steps) == NC_OK && steps == 0, "no rows");
    fake::fail_malloc_from = ~(size_t)0;
    check(nc_record_raster(net, 70) == NC_OK && nc_run(net, 2) == NC_OK && fake::faults == 0, "made later");
    nc_destroy(net);
}

// Detectors' tables are on the device before they are read.
static void detectors_order()
{
    for (int delay : {0, 1, 2, 5, 1000}) {
        fake::legacy_delay = delay;
        Made m(40, 100);
        nc_net* net = m.create();
        const float at[6] = {1, 1, 1, 0.5f, 1, 1.5f}, radius[2] = {9, 9};
        float v[2] = {0, 0};
        check(nc_set_detectors(net, 2, at, radius) == NC_OK, "set");
        check(nc_get_detector_voltages(net, v, 2, nullptr) == NC_OK && v[0] == -70.0f && v[1] == -70.0f,
              "voltages, delay " + std::to_string(delay));
        nc_destroy(net);
    }
    check(fake::faults == 0, "neurons out of range");
}

// Detectors that cannot be added for want of memory leave the ones before them.
static void detectors_refused()
{
    const float at[3] = {1, 1, 1}, radius[1] = {9};
    for (int64_t call = 0; call < 2; ++call) {
        Made m(40, 100);
        nc_net* net = m.create();
        for (int round = 0; round < 2; ++round) {
            float v[2] = {0, 0};
            int32_t count = -1;
            fake::fail_malloc_at = fake::mallocs + call;
            check(nc_set_detectors(net, 1, at, radius) == NC_ERR_CUDA, "refused");
            fake::fail_malloc_at = -1;
            check(nc_get_detector_voltages(net, v, 2, &count) == NC_OK && count == round, "as many as before");
            check(fake::faults == 0 && v[0] == (round ? -70.0f : 0.0f), "voltages");
            check(nc_set_detectors(net, 1, at, radius) == NC_OK, "added later");
        }
        const size_t held = fake::held;
        nc_destroy(net);
        check(held > 0 && fake::held == 0, "memory given back");
    }
}

// Every read-back of a network's results, once.
static bool reads(nc_net* net, const Made& m)
{
    std::vector<float> w(m.w.size()), per(2 * (size_t)m.n);
    std::vector<int32_t> d(m.w.size());
    std::vector<uint8_t> inh(m.w.size()), rows(4 * (((size_t)m.n + 7) / 8));
    std::vector<nc_synapse_snapshot> snap(m.w.size());
    int64_t count = 0;
    int32_t steps = 0;
    nc_stats st;
    return nc_read_weights(net, w.data()) == NC_OK && m.same(w) && nc_read_potentials(net, per.data()) == NC_OK &&
           nc_read_potact(net, per.data()) == NC_OK && nc_read_last_fire(net, per.data()) == NC_OK &&
           nc_read_delays(net, d.data()) == NC_OK && nc_read_inhibitory(net, inh.data()) == NC_OK &&
           nc_read_raster(net, rows.data(), (int64_t)rows.size(), &steps) == NC_OK &&
           nc_read_synapse_snapshots(net, snap.data(), (int64_t)snap.size(), &count) == NC_OK &&
           nc_get_stats(net, &st) == NC_OK;
}

// A read-back allocates no device memory, the first one neither.
static void reads_allocate_nothing()
{
    for (int mode : {NC_STEP_DENSE, NC_STEP_EVENT, NC_STEP_AUTO}) {
        Made m(200, 3000, mode);
        nc_net* net = m.create();
        check(nc_record_raster(net, 4) == NC_OK && nc_run_noalloc(net, 4, nullptr) == NC_OK, "run");
        const int64_t calls = fake::mallocs;
        const size_t held = fake::held;
        check(reads(net, m), std::string("reads: ") + nc_last_error());
        check(fake::mallocs == calls && fake::held == held, "allocations in the reads of form " + std::to_string(mode));
        nc_destroy(net);
    }
    Made a(200, 3000), b(31, 90);
    nc_net_spec specs[2] = {a.spec(5), b.spec(9)};
    nc_batch* batch = nullptr;
    check(nc_batch_create(2, specs, &batch) == NC_OK, "batch");
    const int64_t calls = fake::mallocs;
    std::vector<float> got(a.w.size());
    check(nc_batch_read_weights(batch, 0, got.data()) == NC_OK && a.same(got), "first network");
    check(nc_batch_read_weights(batch, 1, got.data()) == NC_OK && b.same(got), "second network");
    check(fake::mallocs == calls, "allocations in the reads of a batch");
    nc_batch_destroy(batch);
    check(fake::held == 0, "memory given back");
}

// Without memory for the weights' index a network is made all the same, and its weights read.
static void no_index()
{
    for (int mode : {NC_STEP_DENSE, NC_STEP_EVENT}) {
        Made m(2000, 100000, mode);  // (its index is too large for a block of small arrays)
        int64_t before = fake::mallocs;
        nc_destroy(m.create());
        const int64_t calls = fake::mallocs - before;
        fake::fail_malloc_at = fake::mallocs + calls - 1;
        nc_net* net = m.create();
        fake::fail_malloc_at = -1;
        before = fake::mallocs;
        check(net && reads(net, m), std::string("reads: ") + nc_last_error());
        check(fake::mallocs == before, "allocations");
        nc_destroy(net);
        nc_net_spec spec = m.spec(5);
        nc_batch* b = nullptr;
        std::vector<float> got(m.w.size());
        fake::fail_malloc_at = fake::mallocs + calls - 1;
        check(nc_batch_create(1, &spec, &b) == NC_OK, "batch");
        fake::fail_malloc_at = -1;
        check(nc_batch_read_weights(b, 0, got.data()) == NC_OK && m.same(got), "batch weights");
        nc_batch_destroy(b);
    }
}

// A read-back whose kernel cannot be launched leaves the caller's buffer as it was.
static void failed_read()
{
    for (int32_t synapses : {300, 40000, 200000}) {  // one page, several, more than are written directly
        Made m(1000, synapses);
        nc_net* net = m.create();
        std::vector<float> old(m.w.size()), got(m.w.size());
        for (size_t k = 0; k < old.size(); ++k) old[k] = got[k] = -1.0f - (float)k;
        fake::gathers_to_fail = 1;
        check(nc_read_weights(net, got.data()) == NC_ERR_CUDA, "reported");
        check(got == old, "contents, " + std::to_string(synapses) + " synapses");
        check(nc_read_weights(net, got.data()) == NC_OK && m.same(got), "read later");
        nc_destroy(net);
    }
}

// Submits `count` requests, waits for all, and returns their outcomes in the order they came.
static std::vector<nc_request_done> served(nc_server* s, Made& m, int count)
{
    std::vector<int64_t> ids((size_t)count);
    for (int q = 0; q < count; ++q) {
        const nc_net_spec spec = m.spec(5 + 7 * q);
        check(nc_server_submit(s, &spec, &ids[(size_t)q]) == NC_OK, "submit");
    }
    check(nc_server_drain(s) == NC_OK, "drain");
    std::vector<nc_request_done> got((size_t)count + 1), out;
    int32_t n = 0;
    check(nc_server_poll(s, got.data(), count + 1, &n) == NC_OK && n == count, "one outcome a request");
    for (int64_t id : ids)
        for (int32_t k = 0; k < n; ++k)
            if (got[(size_t)k].request_id == id) out.push_back(got[(size_t)k]);
    return out;
}

static nc_server* server(int mode)
{
    nc_server_config c{};
    c.memory_budget_bytes = 32 << 20;
    c.max_networks = 2;
    c.steps_per_batch = 4;
    c.build_threads = 2;
    c.keep_results = 1;
    c.step_mode = mode;
    nc_server* s = nullptr;
    check(nc_server_create(&c, &s) == NC_OK, std::string("server: ") + nc_last_error());
    return s;
}

// A request whose results cannot be read finishes with the error; the others go on.
static void server_read_fails()
{
    for (int mode : {NC_STEP_DENSE, NC_STEP_EVENT}) {
        Made m(60, 500, mode);
        nc_server* s = server(mode);
        fake::gathers_to_fail = 1;
        int failed = 0;
        for (const nc_request_done& d : served(s, m, 5)) {
            std::vector<float> w(m.w.size()), pot((size_t)m.n);
            const int rc = nc_server_fetch(s, d.request_id, w.data(), pot.data());
            if (d.status == NC_OK) check(rc == NC_OK && m.same(w) && pot[0] == -70.0f, "results");
            else check(d.status == NC_ERR_CUDA && rc == NC_ERR_INVALID, "error");
            failed += d.status != NC_OK;
        }
        check(failed == 1, "one failure");
        nc_server_stats st;
        check(nc_server_get_stats(s, &st) == NC_OK && st.finished == 5 && st.resident_bytes == 0, "counts");
        nc_server_destroy(s);
    }
}

// When the device is lost every request, early and late, finishes with the error.
static void server_device_lost()
{
    Made m(60, 500);
    nc_server* s = server(NC_STEP_DENSE);
    for (const nc_request_done& d : served(s, m, 3)) check(d.status == NC_OK, "before");
    fake::graphs_to_fail = 1 << 30;
    for (int round = 0; round < 2; ++round)
        for (const nc_request_done& d : served(s, m, 5)) check(d.status == NC_ERR_CUDA, "after");
    nc_server_stats st;
    check(nc_server_get_stats(s, &st) == NC_OK && st.finished == 13 && st.resident_bytes == 0, "counts");
    nc_server_destroy(s);
    fake::graphs_to_fail = 0;
    check(fake::held == 0, "memory given back");
}

// A small network takes little device memory.
static void footprint()
{
    for (int mode : {NC_STEP_DENSE, NC_STEP_EVENT, NC_STEP_AUTO}) {
        Made few(3, 2, mode), more(1000, 50000, mode);
        nc_net* a = few.create();
        check(fake::held <= 160 << 10, "three neurons: " + std::to_string(fake::held));
        nc_destroy(a);
        a = more.create();
        // some 20 bytes a position dense, 40 event, and what is left of the last blocks
        check(fake::held <= (size_t)(mode == NC_STEP_DENSE ? 4 : 7) << 20, "50,000 synapses: " + std::to_string(fake::held));
        nc_destroy(a);
    }
}

// The dense step's tiles: every quad of every network once and in order, runs of 8 neurons whole
// or split over consecutive blocks, no more tiles than a server has room for.
static void row_plan()
{
    unsigned seed = 1;
    auto rnd = [&](int n) { return (int)((seed = seed * 1664525u + 1013904223u) >> 8) % n; };
    int splits_seen = 0;
    for (int trial = 0; trial < 300; ++trial) {
        std::vector<nc::NetHost> hosts((size_t)(1 + rnd(4)));
        std::vector<nc::RowNet> nets;
        int64_t syn = 0, words = 0;
        int32_t neurons = 0;
        for (size_t q = 0; q < hosts.size(); ++q) {
            nc::NetHost& h = hosts[q];
            h.n = rnd(5) ? 1 + rnd(300) : 8 * rnd(20);
            h.in_ptr.assign(1, 0);
            for (int32_t j = 0; j < h.n; ++j) {
                const int64_t fan = rnd(40) ? rnd(60) : rnd(3) ? 1000 + rnd(3000) : 20000 + rnd(60000);
                const int64_t a = nc::row_align(j), end = h.in_ptr.back() + fan;
                h.in_ptr.push_back((end + a - 1) / a * a);
            }
            h.sp = h.in_ptr.back();
            nets.push_back({&h, (int32_t)q, syn, neurons, neurons + (int32_t)q});
            syn += (h.sp + 31) / 32 * 32;
            neurons += h.n;
            words += (h.n + 31) / 32;
        }
        const int blocks = 1 + rnd(trial % 2 ? 1216 : 40);
        std::vector<NcRowTile> tiles;
        std::vector<int32_t> start;
        nc::plan_rows(nets, blocks, tiles, start);
        check((int)start.size() == blocks + 1 && start[0] == 0 && start[(size_t)blocks] == (int32_t)tiles.size(), "starts");
        check((int64_t)tiles.size() <= words + 2 * blocks, "number of tiles");
        size_t k = 0;
        for (size_t q = 0; q < nets.size(); ++q) {
            const nc::NetHost& h = hosts[q];
            int64_t quad = nets[q].syn_base / 4;
            for (int32_t f = 0; f < h.n;) {
                check(k < tiles.size(), "tiles end early");
                if (k >= tiles.size()) return;
                const NcRowTile first = tiles[k];
                check(first.first == f && first.first % 8 == 0 && first.count > 0 && first.count <= NC_TILE_ROWS, "neurons");
                check(first.neuron == nets[q].neuron_base + f && first.ptr == nets[q].ptr_base + f, "bases");
                const int parts = first.part ? first.part >> 16 : 1;
                check(!first.part || (parts > 1 && first.count <= 8 && (first.part & 0xffff) <= blocks), "part");
                for (int p = 0; p < parts; ++p, ++k) {
                    const NcRowTile& t = tiles[k];
                    check(t.net == (int32_t)q && t.q0 == quad && t.part == first.part && t.count == first.count &&
                              t.first == f && (parts == 1 || t.nq > 0),
                          "quads");
                    quad += t.nq;
                }
                splits_seen += parts > 1;
                f += first.count;
                check(quad == (nets[q].syn_base + h.in_ptr[(size_t)f]) / 4, "rows of the neurons");
            }
        }
        check(k == tiles.size(), "tiles left");
        for (int b = 0; b < blocks; ++b) {
            check(start[(size_t)b] <= start[(size_t)b + 1], "blocks in order");
            for (int32_t t = start[(size_t)b] + 1; t < start[(size_t)b + 1]; ++t)
                check(!tiles[(size_t)t].part || tiles[(size_t)t].part != tiles[(size_t)t - 1].part ||
                          tiles[(size_t)t].net != tiles[(size_t)t - 1].net, "one part of a run to a block");
        }
        if (fails) return;
    }
    check(splits_seen > 100, "runs were split");
}

// A step of the event form after a flush that no call has waited for waits for it as a whole.
static void flush_then_step()
{
    for (int32_t synapses : {0, 300}) {
        Made m(40, synapses, NC_STEP_EVENT);
        nc_net* net = m.create();
        std::vector<nc_synapse_snapshot> snap((size_t)synapses + 1);
        int64_t count = 0;
        for (int round = 0; round < 2; ++round) {
            check(nc_run(net, 3) == NC_OK, "run");
            check(nc_read_synapse_snapshots(net, snap.data(), synapses + 1, &count) == NC_OK, "snapshots");
            check(nc_run_noalloc(net, 1, nullptr) == NC_OK, "step");
        }
        check(fake::early_steps == 0, "steps that may be early, " + std::to_string(synapses) + " synapses");
        nc_destroy(net);
    }
}

int main(int argc, char** argv)
{
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "weights_order") weights_order();
    else if (what == "raster_order") raster_order();
    else if (what == "raster_refused") raster_refused();
    else if (what == "detectors_order") detectors_order();
    else if (what == "detectors_refused") detectors_refused();
    else if (what == "reads_allocate_nothing") reads_allocate_nothing();
    else if (what == "no_index") no_index();
    else if (what == "failed_read") failed_read();
    else if (what == "server_read_fails") server_read_fails();
    else if (what == "server_device_lost") server_device_lost();
    else if (what == "footprint") footprint();
    else if (what == "row_plan") row_plan();
    else if (what == "flush_then_step") flush_then_step();
    else check(false, "no such check: " + what);
    std::printf("%s\n", fails ? "FAILED" : "OK");
    return fails != 0;
}
