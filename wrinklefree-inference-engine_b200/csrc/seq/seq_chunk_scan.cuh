// The scan of one block (seq_chunk.cu): no header but the text of a kernel and of a function.  As the body of the kernel it keeps the registers that it had there; as a
// function that the kernel calls, inlined, two column tiles without the correction took 162 in place of 150 (8 % of the time: matrix memory, 20 heads of 128 x 128, one
// portion of 600 tokens 180 us, 167 so), with a decay per row 168 and 12 bytes spilled in place of 153.
    using L = CrStage<DS, VEC, DELTA>;
    constexpr int REC = cr_rec_floats(DS, VEC), NT = DS / (8 * CR_WARPS), STEP = CR_THREADS / (DS / 4);
    constexpr int PARTS = DELTA ? 2 * CT : 2;              // partial sums of a warp: S^T q of each column tile, then R of each
    extern __shared__ __align__(16) float sm[];
    float* red = sm + 2 * L::FLOATS;                      // [4 warps][PARTS][16 columns][CR_RS]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int col0 = tile0 * CR_COLS, dvs = D.dv + D.ones_col, kh = h / (D.H / D.Hk);
    const int first = seg * SCAN_CHUNK, seq0 = b.seq_start[sq], start = seq0 + first;
    const int len = sg.pass ? min(SCAN_CHUNK, b.seq_len[sq] - first) : b.seq_len[sq], nch = (len + CR - 1) / CR;
    if (len <= 0) return;                                 // this sequence has fewer segments
    const size_t entry = ((size_t)(seq0 / SCAN_CHUNK + sq + seg) * D.H + h) * D.d * dvs;
    const float* S0 = sg.pass == 3 ? sg.start + entry : state + (size_t)b.seq_slot[sq] * slot_stride + (size_t)h * D.d * dvs;
    const float* rec0 = w.rec + ((size_t)(seq0 / CR + sq + first / CR) * D.H + h) * REC;
    float prod = 1.f;
    const int row0 = warp * 8 * NT;                       // this warp's key rows
    // s[ct][nt]: columns col0 + 16 ct + g (0, 1) and + 8 (2, 3), rows row0 + 8 nt + 2 t (0, 2) and + 1 (1, 3)
    float s[CT][NT][4];
    auto at_state = [&](int ct, int nt, int e, bool& ok) -> size_t {
        const int r = row0 + 8 * nt + 2 * t + (e & 1), c = col0 + 16 * ct + g + 8 * (e >> 1);
        ok = r < D.d && c < dvs;
        return (size_t)r * dvs + c;
    };
#pragma unroll
    for (int ct = 0; ct < CT; ++ct)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) { bool ok; const size_t i = at_state(ct, nt, e, ok); s[ct][nt][e] = ok && sg.pass != 1 ? S0[i] : 0.f; }
    auto stage = [&](int ch) {
        float* dst = sm + (ch & 1) * L::FLOATS;
        const float* src = rec0 + (size_t)ch * D.H * REC;
        if (tid < 64) {
            const int r = tid >> 2, c = (tid & 3) * 4;
            if (DELTA) cr_cp16(dst + L::T + r * L::TS + c, src + r * CR + c);
            cr_cp16(dst + L::B + r * L::TS + c, src + 256 + r * CR + c);
        }
        const int c = (tid % (DS / 4)) * 4, r0 = tid / (DS / 4);
        if (VEC) {
            const float* x = src + 512 + r0 * DS + c;
#pragma unroll
            for (int r = 0; r < CR; r += STEP, x += STEP * DS) {
                if (sg.pass != 1) cr_cp16(dst + L::Q + (r0 + r) * L::QS + c, x);
                if (DELTA) cr_cp16(dst + L::K + (r0 + r) * L::QS + c, x + CR * DS);
                cr_cp16(dst + L::N + (r0 + r) * L::KS + c, x + 2 * CR * DS);
            }
            if (tid < DS / 4) cr_cp16(dst + L::G + tid * 4, src + 512 + 3 * CR * DS + tid * 4);
        } else {
            const float* row = w.qkv + (size_t)(start + ch * CR + r0) * w.ld + kh * D.d + c;
            const int left = c < D.d ? len - ch * CR - r0 : 0;
#pragma unroll
            for (int r = 0; r < CR; r += STEP, row += (size_t)STEP * w.ld) {
                float *qd = dst + L::Q + (r0 + r) * L::QS + c, *kd = dst + L::K + (r0 + r) * L::QS + c, *nd = dst + L::N + (r0 + r) * L::KS + c;
                if (r < left) {
                    if (sg.pass != 1) cr_cp16(qd, row + w.q_off);
                    if (DELTA) cr_cp16(kd, row + w.k_off);
                    cr_cp16(nd, row + w.k_off);
                } else {
                    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
                    *reinterpret_cast<float4*>(qd) = z;
                    if (DELTA) *reinterpret_cast<float4*>(kd) = z;
                    *reinterpret_cast<float4*>(nd) = z;
                }
            }
            if (tid < 12) cr_cp16(dst + L::G + tid * 4, src + 512 + tid * 4);
        }
        cp_async_commit();
    };
    // a chunk's values (times beta without the correction), in accumulator layout: columns g and g + 8, tokens 8 n + 2 t and + 1
    float vn[CT][2][4], bn[2][2];
    auto values = [&](int tok0) {
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int tk = tok0 + 8 * n + 2 * t + (e & 1);
#pragma unroll
                for (int ct = 0; ct < CT; ++ct) {
                    const int c = col0 + 16 * ct + g + 8 * (e >> 1);
                    vn[ct][n][e] = tk >= len || c >= dvs ? 0.f : c == D.dv ? 1.f : w.qkv[(size_t)(start + tk) * w.ld + w.v_off + h * D.dv + c];
                }
                if (!DELTA && e < 2) bn[n][e] = w.beta && tk < len ? w.beta[(size_t)(start + tk) * D.H + h] : 1.f;
            }
    };
    float watch[4] = {0.f, 0.f, 0.f, 0.f};
    stage(0);
    values(0);
    for (int ch = 0; ch < nch; ++ch) {
        const int tok0 = ch * CR;
        float v[CT][2][4];
#pragma unroll
        for (int ct = 0; ct < CT; ++ct)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) v[ct][n][e] = DELTA ? vn[ct][n][e] : vn[ct][n][e] * bn[n][e & 1];
        cp_async_wait<0>();
        __syncthreads();                                  // chunk ch has landed; everyone is done with the other half and the partial sums
        if (ch + 1 < nch) { stage(ch + 1); values(tok0 + CR); }
        const float* st = sm + (ch & 1) * L::FLOATS;
        if (DELTA || sg.pass != 1) {
        // ---- this warp's rows' share of S^T q and R; the small terms in accumulators of their own, so that no product waits for the one before it
        float oq[CT][2][4], rk[CT][2][4], oql[CT][2][4], rkl[CT][2][4];
#pragma unroll
        for (int ct = 0; ct < CT; ++ct)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) oq[ct][n][e] = oql[ct][n][e] = rk[ct][n][e] = rkl[ct][n][e] = 0.f;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const int r = row0 + 8 * nt + 2 * t;
            CrB q[2], k[2];
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                q[n] = cr_b2(st + L::Q + (8 * n + g) * L::QS + r);
                if (DELTA) k[n] = cr_b2(st + L::K + (8 * n + g) * L::QS + r);
            }
#pragma unroll
            for (int ct = 0; ct < CT; ++ct) {
                const CrA a = cr_a(s[ct][nt]);
#pragma unroll
                for (int n = 0; n < 2; ++n) { cr_mma(oql[ct][n], a.l, q[n].h); if (DELTA) cr_mma(rkl[ct][n], a.l, k[n].h); }
#pragma unroll
                for (int n = 0; n < 2; ++n) { cr_mma(oq[ct][n], a.h, q[n].h); if (DELTA) cr_mma(rk[ct][n], a.h, k[n].h); }
#pragma unroll
                for (int n = 0; n < 2; ++n) { cr_mma(oql[ct][n], a.h, q[n].l); if (DELTA) cr_mma(rkl[ct][n], a.h, k[n].l); }
            }
        }
        float* mine = red + warp * PARTS * CR_COLS * CR_RS;
#pragma unroll
        for (int ct = 0; ct < CT; ++ct)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    float* to = mine + (ct * CR_COLS + g + 8 * c) * CR_RS + 8 * n + 2 * t;
                    *reinterpret_cast<float2*>(to) = make_float2(oq[ct][n][2 * c] + oql[ct][n][2 * c], oq[ct][n][2 * c + 1] + oql[ct][n][2 * c + 1]);
                    if (DELTA) *reinterpret_cast<float2*>(to + CT * CR_COLS * CR_RS) = make_float2(rk[ct][n][2 * c] + rkl[ct][n][2 * c], rk[ct][n][2 * c + 1] + rkl[ct][n][2 * c + 1]);
                }
        }
        if (DELTA || sg.pass != 1) __syncthreads();
        auto total = [&](int part, int n, int c) {
            const float* p = red + (part * CR_COLS + g + 8 * c) * CR_RS + 8 * n + 2 * t;
            float2 x = *reinterpret_cast<const float2*>(p);
#pragma unroll
            for (int k = 1; k < CR_WARPS; ++k) { const float2 y = *reinterpret_cast<const float2*>(p + k * PARTS * CR_COLS * CR_RS); x.x += y.x; x.y += y.y; }
            return x;
        };
        float u[CT][2][4];
        if (DELTA) {                                      // every warp forms all of U: it is the update's operand
            CrB tb[3];                                    // T is lower triangular
            tb[0] = cr_b2(st + L::T + g * L::TS + 2 * t); tb[1] = cr_b2(st + L::T + (8 + g) * L::TS + 2 * t); tb[2] = cr_b2(st + L::T + (8 + g) * L::TS + 2 * t + 8);
#pragma unroll
            for (int ct = 0; ct < CT; ++ct) {
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        float2 r = total(CT + ct, n, c);
                        if (!VEC) { r.x *= st[L::G + 8 * n + 2 * t]; r.y *= st[L::G + 8 * n + 2 * t + 1]; }
                        v[ct][n][2 * c] -= r.x; v[ct][n][2 * c + 1] -= r.y;
                    }
                const CrA w0 = cr_a(v[ct][0]), w1 = cr_a(v[ct][1]);
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    u[ct][n][0] = u[ct][n][1] = u[ct][n][2] = u[ct][n][3] = 0.f;
                    cr_mma3(u[ct][n], w0, tb[n]);
                    if (n) cr_mma3(u[ct][n], w1, tb[2]);
                }
            }
        } else {
#pragma unroll
            for (int ct = 0; ct < CT; ++ct)
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) u[ct][n][e] = v[ct][n][e];
        }
#pragma unroll
        for (int ct = 0; ct < CT; ++ct)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) cr_watch(watch[2 * n + (e & 1)], u[ct][n][e]);
        if (warp < 2 * CT && sg.pass != 1) {                              // the read-out of 8 tokens of a column tile each
            const int n = warp & 1, ct = warp >> 1;
            float out[4], add[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                float2 x = total(ct, n, c);
                if (!VEC) { x.x *= st[L::G + 8 * n + 2 * t]; x.y *= st[L::G + 8 * n + 2 * t + 1]; }
                out[2 * c] = x.x; out[2 * c + 1] = x.y;
            }
            float ua[2][4];                               // this tile's values: a choice of registers, not an indexed array
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int e = 0; e < 4; ++e) ua[m][e] = CT == 2 && ct ? u[CT - 1][m][e] : u[0][m][e];
            const float* row = st + L::B + (8 * n + g) * L::TS + 2 * t;
            cr_mma3(add, cr_a(ua[0]), cr_b2(row));
            if (n) cr_mma3(add, cr_a(ua[1]), cr_b2(row + 8));
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int tk = tok0 + 8 * n + 2 * t + (e & 1), c = col0 + 16 * ct + g + 8 * (e >> 1);
                if (tk < len && c < dvs) o[((size_t)(start + tk) * D.H + h) * dvs + c] = (out[e] + add[e]) * D.o_scale;
            }
        }
        if (!VEC) prod *= st[L::G + 32];
        // ---- state update: the chunk's own sum from zero, so that the state itself is only ever rounded to nearest (the matrix unit's sums are cut off)
        CrB k0[NT], k1[NT];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const float* kr = st + L::N + 2 * t * L::KS + row0 + 8 * nt + g;
            k0[nt] = cr_b(kr[0], kr[L::KS]); k1[nt] = cr_b(kr[8 * L::KS], kr[9 * L::KS]);
        }
#pragma unroll
        for (int ct = 0; ct < CT; ++ct) {
            if (!VEC) {
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    const float d0 = st[L::G + 16 + 8 * n + 2 * t], d1 = st[L::G + 16 + 8 * n + 2 * t + 1];
                    u[ct][n][0] *= d0; u[ct][n][1] *= d1; u[ct][n][2] *= d0; u[ct][n][3] *= d1;
                }
            }
            const CrA u0 = cr_a(u[ct][0]), u1 = cr_a(u[ct][1]);
            float ds[NT][4];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) ds[nt][0] = ds[nt][1] = ds[nt][2] = ds[nt][3] = 0.f;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) cr_mma(ds[nt], u0.l, k0[nt].h);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) cr_mma(ds[nt], u0.h, k0[nt].l);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) cr_mma(ds[nt], u1.l, k1[nt].h);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) cr_mma(ds[nt], u1.h, k1[nt].l);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) cr_mma(ds[nt], u0.h, k0[nt].h);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) cr_mma(ds[nt], u1.h, k1[nt].h);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                float2 ge;
                if (VEC) ge = *reinterpret_cast<const float2*>(st + L::G + row0 + 8 * nt + 2 * t);
                else ge.x = ge.y = st[L::G + 32];
                s[ct][nt][0] = fmaf(s[ct][nt][0], ge.x, ds[nt][0]); s[ct][nt][1] = fmaf(s[ct][nt][1], ge.y, ds[nt][1]);
                s[ct][nt][2] = fmaf(s[ct][nt][2], ge.x, ds[nt][2]); s[ct][nt][3] = fmaf(s[ct][nt][3], ge.y, ds[nt][3]);
            }
        }
    }
    // a state that has left the finite numbers does not come back: looked at once
#pragma unroll
    for (int ct = 0; ct < CT; ++ct)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) cr_watch(watch[e], s[ct][nt][e]);
    const int lost = __syncthreads_or(!((watch[0] + watch[1]) + (watch[2] + watch[3]) == 0.f));
    int* mark = w.redo + ((size_t)sq * D.H + h) * w.cols + tile0;      // the preparation marks all of a head's tiles
    const int tiles = min(CT, w.cols - tile0);
    if (lost && tid < tiles) mark[tid] = 1;
    if (sg.pass == 3) return;                             // scan_prefix_kernel has left the end states
    if (sg.pass == 0 && (lost || *mark)) return;          // the slot keeps the start state for chunk_redo_kernel
    float* S1 = sg.pass ? sg.local + entry : state + (size_t)b.seq_slot[sq] * slot_stride + (size_t)h * D.d * dvs;
#pragma unroll
    for (int ct = 0; ct < CT; ++ct)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) { bool ok; const size_t i = at_state(ct, nt, e, ok); if (ok) S1[i] = s[ct][nt][e]; }
    if (!VEC && sg.pass && tile0 == 0 && tid == 0) sg.prod[(size_t)(seq0 / SCAN_CHUNK + sq + seg) * D.H + h] = prod;
