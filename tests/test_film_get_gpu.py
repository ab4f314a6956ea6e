"""lts_film_get without a film of the loaded scene."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_film_of_a_smaller_scene_is_not_read(built_lib, tmp_path):
    """After a render at 32 x 32 and the load of a 96 x 64 film, nothing has been rendered for the film that
    lts_film_get would copy; a render at the new size makes it."""
    import lighttransportsimulation_gb300 as lts
    from lighttransportsimulation_gb300 import scenes
    sc, sub = scenes.write_box_sphere(str(tmp_path), level=1)
    ctx = lts.Context(0)
    film = np.zeros(96 * 64 * 3, np.float32)
    ptr = film.ctypes.data_as(ctypes.c_void_p)
    s = lts.Scene.parse(ctx, str(tmp_path), sc, sub, 32, 32)
    lts.PathTracingIntegrator(2, 3, s).render(1, 1)
    s = lts.Scene.parse(ctx, str(tmp_path), sc, sub, 96, 64)
    assert ctx.lib.lts_film_get(ctx.h, ptr, None) != 0
    assert "nothing rendered" in ctx.lib.lts_last_error(ctx.h).decode() and not film.any()
    want = lts.PathTracingIntegrator(2, 3, s).render(1, 1)["film"]
    assert ctx.lib.lts_film_get(ctx.h, ptr, None) == 0
    assert np.array_equal(film.reshape(want.shape), want)
    ctx.close()
