/* Steps of the same sessions keep their work list on the device.  Here the
 * arena that holds it is grown twice between two steps and the second time
 * gets its first addresses back (in host and in device memory), whose contents
 * are gone: the next steps still have to run on the right list.  The engine's
 * host code on a stand-in for the CUDA runtime (fake_cuda.h). */
#include "fake_cuda.h"

#include "engine.cu"

static int steps_run;
static std::vector<const void *> desc_host, desc_dev;   /* the descriptor arenas, by step slot */

extern "C" int64_t h261b_bits_slot_bytes(int32_t, int32_t) { return 0; }
extern "C" h261b_bits_layout_t h261b_bits_layout(int32_t, int32_t) { return h261b_bits_layout_t{}; }
extern "C" int h261b_launch_ratectrl(h261b_session_dev_t *, int32_t, void *) { return 0; }
extern "C" int h261b_launch_bitstream(h261b_session_dev_t *, int32_t, const uint32_t *, int32_t, h261b_step_dev_t *,
                                      uint8_t *, int64_t, int32_t, int32_t, void *, void *, int32_t)
{
    return 0;
}
extern "C" int h261b_launch_fetch(void *dst0, const void *src0, int64_t bytes0, void *dst1, const void *src1,
                                  int64_t bytes1, void *zero, int64_t zero_bytes, int32_t, void *)
{
    memcpy(dst0, src0, (size_t)bytes0);
    memcpy(dst1, src1, (size_t)bytes1);
    if (zero_bytes)
        memset(zero, 0, (size_t)zero_bytes);
    desc_host.push_back(src0);
    desc_dev.push_back(dst0);
    return 0;
}
extern "C" int h261b_launch_step(const h261b_session_dev_t *sessions, const uint32_t *work, int32_t n_work, int32_t,
                                 int32_t, int32_t, int32_t *, void *)
{
    int32_t at = 0;
    for (uint32_t k = 0; at < n_work; k++)
        for (uint32_t m = 0; m < (uint32_t)(sessions[k].mbw * sessions[k].mbh); m++, at++)
            CHECK_THAT(at < n_work && work[at] == (k << 12 | m), "step %d: work item %d is %08x", steps_run, at,
                       work[at]);
    steps_run++;
    return 0;
}

int main()
{
    h261b_engine_config_t c;
    h261b_engine_config_default(&c);
    c.copy_threads = 1;
    c.warps_per_cta = 8;   /* one launch a step */
    c.kernel_split = c.tail_items = c.staging = 1;
    h261b_engine_t *e = nullptr;
    CHECK_THAT(h261b_engine_create(&c, &e) == 0, "create: %s", h261b_last_error());
    h261b_session_config_t sc = {};
    sc.width = 176;
    sc.height = 144;
    sc.quant = 8;
    std::vector<int32_t> ids(3);
    for (int32_t &id : ids)
        CHECK_THAT(h261b_session_open(e, &sc, &id) == 0, "open: %s", h261b_last_error());
    std::vector<uint8_t> pic(176 * 144, 1);
    auto step = [&] {
        for (int32_t id : ids)
            CHECK_THAT(h261b_session_submit(e, id, pic.data(), pic.data(), pic.data(), 0) == 0, "submit");
        CHECK_THAT(h261b_engine_step(e) == 3 && h261b_engine_sync(e) == 0, "step: %s", h261b_last_error());
    };
    for (int i = 0; i < 6; i++)
        step();
    const std::vector<const void *> host(desc_host.end() - 3, desc_host.end()), dev(desc_dev.end() - 3, desc_dev.end());
    /* the arenas grow out of the way, then once more: of this growth the
     * descriptor arenas are the small blocks, in the order of the slots, and
     * each gets the addresses that its slot began with */
    int top = kSlots;
    fake_pick = [&](size_t, bool) { return fake_base + kSlot * --top; };
    CHECK_THAT(h261b_engine_reserve_step(e, &sc, 2000) == 0, "reserve: %s", h261b_last_error());
    size_t nh = 0, nd = 0;
    fake_pick = [&](size_t bytes, bool pinned) -> void * {
        return bytes >= (size_t)16 << 20 ? fake_base + kSlot * --top : (void *)(pinned ? host[nh++] : dev[nd++]);
    };
    CHECK_THAT(h261b_engine_reserve_step(e, &sc, 2000) == 0, "reserve: %s", h261b_last_error());
    fake_pick = nullptr;
    CHECK_THAT(nh == 3 && nd == 3, "%zu and %zu small blocks", nh, nd);
    for (int i = 0; i < 6; i++)
        step();
    for (int i = 0; i < 3; i++)
        CHECK_THAT(desc_host[desc_host.size() - 3 + i] == host[i] && desc_dev[desc_dev.size() - 3 + i] == dev[i],
                   "the arenas are not where the test put them");
    CHECK_THAT(h261b_engine_destroy(e) == 0, "destroy");
    CHECK_THAT(steps_run == 12, "%d steps", steps_run);
    puts("ok");
    return 0;
}
