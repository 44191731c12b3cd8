// A resident pass whose wait runs out: one block's messages to a neighbour go to a mailbox that nobody
// reads (inside the exchange buffer), so that the neighbour gives up after its time limit and the others
// with it.  The pass must end by itself with the status, and with the tables as they were the plan must
// give its first results again.  Arguments: nx nz CPML double(0/1) the widest block's columns a thread.
// Prints "ok".
#include "rtm_engine.cu"

static int bad(const char *what)
{
    printf("%s (%s)\n", what, rtm_last_error());
    return 1;
}

int main(int argc, char **argv)
{
    if (argc != 6) return bad("arguments");
    rtm_params p;
    memset(&p, 0, sizeof p);
    rtm_params_defaults(&p);
    p.nx = atoi(argv[1]); p.nz = atoi(argv[2]);
    p.th_left = p.th_right = p.th_up = p.th_down = atoi(argv[3]);
    p.compute = atoi(argv[4]) ? RTM_COMPUTE_FP64 : RTM_COMPUTE_FP32;
    p.dx = 10.0f; p.dt = 1e-3f; p.nt = 40; p.n_wavelet = 20; p.shot_x = p.nx / 2; p.shot_z = 2;
    p.rec_spacing = 2; p.rec_count = p.nx; p.rec_depth = 2; p.time_slices = 4;
    rtm_plan *P = nullptr;
    if (rtm_plan_create(&p, &P) != RTM_OK) return bad("create");
    const int want = atoi(argv[5]);
    if (P->res[0].cw != want) { printf("%d columns a thread, not %d\n", P->res[0].cw, want); return 1; }
    const size_t nv = (size_t)P->g.dimx * P->g.dimz, ns = (size_t)p.rec_count * p.nt, ni = (size_t)p.nx * p.nz;
    std::vector<float> vel(nv, 2000.0f), wav(p.n_wavelet), seis(ns);
    for (size_t k = 0; k < wav.size(); ++k) wav[k] = (float)(k % 7) * 0.1f;
    for (size_t k = 0; k < ns; ++k) seis[k] = (float)((k * 2654435761u) % 1000) * 1e-3f - 0.5f;
    float *d_vel, *d_wav, *d_seis;
    if (cudaMalloc(&d_vel, nv * 4) || cudaMalloc(&d_wav, wav.size() * 4) || cudaMalloc(&d_seis, ns * 4)) return bad("malloc");
    cudaMemcpy(d_vel, vel.data(), nv * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(d_wav, wav.data(), wav.size() * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(d_seis, seis.data(), ns * 4, cudaMemcpyHostToDevice);
    double *d_img;
    if (cudaMalloc(&d_img, ni * sizeof(double))) return bad("malloc");
    auto migrate = [&](std::vector<double> &img) {
        img.assign(ni, 0.0);
        int st = rtm_plan_forward(P, d_vel, d_wav, nullptr);
        if (st == RTM_OK) st = rtm_plan_sync(P);
        if (st == RTM_OK) st = rtm_plan_adjoint(P, d_seis, nullptr, nullptr);
        if (st == RTM_OK) st = rtm_plan_read_image(P, 0, 1, d_img);
        if (st == RTM_OK) st = rtm_plan_sync(P);
        cudaMemcpy(img.data(), d_img, ni * sizeof(double), cudaMemcpyDeviceToHost);
        return st;
    };
    std::vector<double> first, again;
    if (migrate(first) != RTM_OK) return bad("first migration");
    // an exchange buffer twice as long, whose second half nobody reads
    const size_t quads = P->xch_bytes / (4 * 2 * P->es);
    unsigned long long *longer = nullptr, *own = P->xch;
    if (cudaMalloc(&longer, 2 * P->xch_bytes) || cudaMemset(longer, 0, 2 * P->xch_bytes)) return bad("malloc");
    for (int back = 0; back < 2; ++back) {
        const int n = P->res[back].nctas;
        std::vector<ResCta> c(n), t;
        ResCta *dev = const_cast<ResCta *>(P->res[back].ctas);
        cudaMemcpy(c.data(), dev, n * sizeof(ResCta), cudaMemcpyDeviceToHost);
        t = c;
        int side = 0;
        while (side < 4 && t[n / 2].dout[side] == 0) ++side;
        if (side == 4) return bad("a block without neighbours");
        t[n / 2].out_off[side] += (unsigned)quads;
        P->xch = longer;
        cudaMemcpy(dev, t.data(), n * sizeof(ResCta), cudaMemcpyHostToDevice);
        cudaMemset(longer, 0, 2 * P->xch_bytes);
        cudaDeviceSynchronize();
        const auto t0 = std::chrono::steady_clock::now();
        const int st = migrate(again);
        const double s = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        if (st != RTM_ERR_TIMEOUT || !strstr(rtm_last_error(), "exchange")) return bad("the lost message went unnoticed");
        if (s < 1.0 || s > 10.0) { printf("gave up after %.1f s\n", s); return 1; }
        cudaMemcpy(dev, c.data(), n * sizeof(ResCta), cudaMemcpyHostToDevice);
        P->xch = own;
        if (migrate(again) != RTM_OK) return bad("migration after it");
        if (memcmp(first.data(), again.data(), ni * sizeof(double)) != 0) return bad("another image after it");
    }
    double most = 0.0;
    for (double v : first) most = std::max(most, std::fabs(v));
    if (!(most > 0.0)) return bad("an empty image");
    rtm_plan_destroy(P);
    if (cudaDeviceSynchronize() != cudaSuccess) return bad("device");
    printf("ok\n");
    return 0;
}
