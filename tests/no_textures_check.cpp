/* The boundary's calls that launch kernels are refused, with a status and
 * without a launch or a copy, when the picture memory is not there: before
 * h261_gpu_device_init_textures, after h261_gpu_device_deinit_textures, and
 * when a part of it could not be allocated.  The boundary's host code on a
 * stand-in for the CUDA runtime (fake_cuda.h). */
#include "fake_cuda.h"

#include "compat.cu"

static int launches;
void h261b::set_error(const char *, ...) {}
extern "C" int h261b_launch_team_picture(const h261b_session_dev_t *d, int32_t, void *)
{
    CHECK_THAT(fake_is_block(d->cur_y) && fake_is_block(d->ref_y) && fake_is_block(d->rec_y), "no picture memory");
    launches++;
    return 0;
}
extern "C" int h261b_launch_step(const h261b_session_dev_t *, const uint32_t *, int32_t, int32_t, int32_t, int32_t,
                                 int32_t *, void *)
{
    CHECK_THAT(false, "not a launch of this size");
    return 0;
}

int main()
{
    const int32_t w = 176, h = 144, n = (w / 16) * (h / 16);
    std::vector<h261_mb_mode_decision_t> mds((size_t)n);
    memset(mds.data(), 0, mds.size() * sizeof(mds[0]));
    for (auto &m : mds)
        m.i_mb_type = H261B_MB_TYPE_INTRA;
    h261_mode_decision_t md = {};
    md.i_mb_width = w / 16;
    md.i_mb_height = h / 16;
    md.prgs_mb = mds.data();
    h261_context_t ctx = {};
    ctx.ps_mode_decision = &md;
    ctx.s_picture.i_quantiser = 8;
    me_gpu_t *me = nullptr;
    std::vector<uint8_t> plane((size_t)w * h, 7);

    auto calls = [&](const char *when, bool taken) {
        const int before = launches;
        int status[4];
        auto reset = [] { g.status = H261B_OK; };
        reset();
        h261_gpu_device_set_current(plane.data(), w, h);
        status[0] = h261b_abi_last_status();
        reset();
        h261_gpu_device_me(me);
        status[1] = h261b_abi_last_status();
        reset();
        h261_gpu_device_encode_macroblocks(&ctx);
        status[2] = h261b_abi_last_status();
        reset();
        h261_gpu_device_decode_macroblocks(&ctx);
        status[3] = h261b_abi_last_status();
        for (int s : status)
            CHECK_THAT((s == H261B_OK) == taken, "%s: %d %d %d %d", when, status[0], status[1], status[2], status[3]);
        CHECK_THAT(launches - before == (taken ? 2 : 0), "%s: %d launches", when, launches - before);
    };

    h261_gpu_init();
    h261_gpu_device_init_me(&me, w, h);
    CHECK_THAT(me, "motion estimation state");
    calls("before the textures", false);
    h261_gpu_device_init_textures(w, h);
    h261_init_macroblocks(&ctx.ps_macroblocks, w, h, 5);
    CHECK_THAT(ctx.ps_macroblocks, "macroblocks");
    calls("with the textures", true);
    h261_gpu_device_deinit_textures();
    calls("after the textures", false);
    h261_gpu_device_init_textures(w, h);
    calls("with new textures", true);
    /* each of the four blocks in turn is refused */
    for (int k = 0; k < 4; k++) {
        fake_fail_after = k;
        h261_gpu_device_init_textures(w, h);
        fake_fail_after = -1;
        calls("with a part of the textures", false);
    }
    h261_gpu_device_init_textures(w, h);
    calls("with textures again", true);
    /* a picture larger than the macroblock state's host arrays */
    h261_gpu_device_init_textures(2 * w, 2 * h);
    g.status = H261B_OK;
    ctx.ps_macroblocks->pui8_reconstructed_Y_host[(size_t)n * 256 - 1] = 99;
    h261_gpu_device_decode_macroblocks(&ctx);
    CHECK_THAT(h261b_abi_last_status() == H261B_ERR_ARG, "a picture of another size was decoded");
    CHECK_THAT(ctx.ps_macroblocks->pui8_reconstructed_Y_host[(size_t)n * 256 - 1] == 99, "and written");
    h261_deinit_macroblocks(ctx.ps_macroblocks);
    h261_gpu_device_deinit_me(&me);
    h261_gpu_device_deinit_textures();
    puts("ok");
    return 0;
}
