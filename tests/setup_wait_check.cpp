/* What the set-up writes by copies and clears on the legacy stream, which CUDA
 * lets outlive their call, is in device memory before a stream that does not
 * wait for the legacy stream uses it: the engine's work counters and the
 * boundary's work list of a large picture.  The host code of both on a stand-in
 * for the CUDA runtime (fake_cuda.h). */
#include "fake_cuda.h"

#include "engine.cu"
#undef CK
#include "compat.cu"

static int launches;

extern "C" int64_t h261b_bits_slot_bytes(int32_t, int32_t) { return 0; }
extern "C" h261b_bits_layout_t h261b_bits_layout(int32_t, int32_t) { return h261b_bits_layout_t{}; }
extern "C" int h261b_launch_ratectrl(h261b_session_dev_t *, int32_t, void *) { return 0; }
extern "C" int h261b_launch_bitstream(h261b_session_dev_t *, int32_t, const uint32_t *, int32_t, h261b_step_dev_t *,
                                      uint8_t *, int64_t, int32_t, int32_t, void *, void *, int32_t)
{
    return 0;
}
extern "C" int h261b_launch_fetch(void *dst0, const void *src0, int64_t bytes0, void *dst1, const void *src1,
                                  int64_t bytes1, void *, int64_t, int32_t, void *)
{
    memcpy(dst0, src0, (size_t)bytes0);
    memcpy(dst1, src1, (size_t)bytes1);
    return 0;
}
extern "C" int h261b_launch_team_picture(const h261b_session_dev_t *, int32_t, void *) { return 0; }
extern "C" int h261b_launch_step(const h261b_session_dev_t *, const uint32_t *work, int32_t n_work, int32_t, int32_t,
                                 int32_t, int32_t *sched, void *)
{
    launches++;
    for (int32_t i = 0; i < n_work; i++)
        CHECK_THAT(work[i] == (uint32_t)i, "work item %d is %08x", i, work[i]);
    for (int i = 0; sched && i < 2; i++)
        CHECK_THAT(sched[i] == 0, "work counter %d is %08x", i, sched[i]);
    return 0;
}

static void check_engine()
{
    h261b_engine_config_t c;
    h261b_engine_config_default(&c);
    c.copy_threads = 1;
    h261b_engine_t *e = nullptr;
    CHECK_THAT(h261b_engine_create(&c, &e) == 0, "create: %s", h261b_last_error());
    h261b_session_config_t sc = {};
    sc.width = sc.height = 64;
    sc.quant = 8;
    int32_t id = 0;
    CHECK_THAT(h261b_session_open(e, &sc, &id) == 0, "open: %s", h261b_last_error());
    std::vector<uint8_t> pic(64 * 64, 1);
    CHECK_THAT(h261b_session_submit(e, id, pic.data(), pic.data(), pic.data(), 0) == 0, "submit");
    CHECK_THAT(h261b_engine_step(e) == 1, "step: %s", h261b_last_error());
    CHECK_THAT(h261b_engine_destroy(e) == 0, "destroy");
}

static void check_boundary()
{
    const int32_t w = 640, h = 480;
    h261_gpu_init();
    h261_gpu_device_init_textures(w, h);
    me_gpu_t *me = nullptr;
    h261_gpu_device_init_me(&me, w, h);
    CHECK_THAT(me && h261b_abi_last_status() == H261B_OK, "set-up");
    h261_gpu_device_me(me);
    CHECK_THAT(h261b_abi_last_status() == H261B_OK, "motion estimation: %s", h261b_last_error());
    h261_gpu_device_deinit_me(&me);
    h261_gpu_device_deinit_textures();
}

int main(int argc, char **argv)
{
    CHECK_THAT(argc == 2, "engine or boundary");
    if (!strcmp(argv[1], "engine"))
        check_engine();
    else
        check_boundary();
    CHECK_THAT(launches >= 1, "nothing was launched");
    puts("ok");
    return 0;
}
