/* A host LAPACK whose zggev reports a failure from its FAIL_AT-th call on and
 * otherwise passes every call to the library REAL_LAPACK names (its symbols
 * with or without the prefix scipy_). */
#include <dlfcn.h>
#include <stdio.h>
#include <stdlib.h>

static void *real(const char *name)
{
    static void *lib;
    char buf[64];
    void *f;
    if (!lib) lib = dlopen(getenv("REAL_LAPACK"), RTLD_NOW | RTLD_LOCAL);
    if (!lib) return NULL;
    snprintf(buf, sizeof buf, "scipy_%s", name);
    f = dlsym(lib, buf);
    return f ? f : dlsym(lib, name);
}

typedef void *P;

void zggev_(P jl, P jr, P n, P a, P lda, P b, P ldb, P al, P be, P vl, P ldvl, P vr, P ldvr, P work, P lwork, P rwork,
            int *info, size_t l1, size_t l2)
{
    static int calls;
    if (++calls >= atoi(getenv("FAIL_AT"))) {
        *info = 3;
        return;
    }
    ((void (*)(P, P, P, P, P, P, P, P, P, P, P, P, P, P, P, P, int *, size_t, size_t))real("zggev_"))(
        jl, jr, n, a, lda, b, ldb, al, be, vl, ldvl, vr, ldvr, work, lwork, rwork, info, l1, l2);
}

void zpotrf_(P uplo, P n, P a, P lda, P info, size_t l)
{
    ((void (*)(P, P, P, P, P, size_t))real("zpotrf_"))(uplo, n, a, lda, info, l);
}

void zgesdd_(P jobz, P m, P n, P a, P lda, P s, P u, P ldu, P vt, P ldvt, P work, P lwork, P rwork, P iwork, P info,
             size_t l)
{
    ((void (*)(P, P, P, P, P, P, P, P, P, P, P, P, P, P, P, size_t))real("zgesdd_"))(
        jobz, m, n, a, lda, s, u, ldu, vt, ldvt, work, lwork, rwork, iwork, info, l);
}

void zgeev_(P jl, P jr, P n, P a, P lda, P w, P vl, P ldvl, P vr, P ldvr, P work, P lwork, P rwork, P info, size_t l1,
            size_t l2)
{
    ((void (*)(P, P, P, P, P, P, P, P, P, P, P, P, P, P, size_t, size_t))real("zgeev_"))(
        jl, jr, n, a, lda, w, vl, ldvl, vr, ldvr, work, lwork, rwork, info, l1, l2);
}
