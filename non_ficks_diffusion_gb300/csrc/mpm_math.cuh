// mpm_math.cuh — precision policies and per-particle 3x3 algebra for the sm_103a kernels:
// quadratic B-spline weights, a 3x3 SVD, fixed-corotated stress, its differential and the
// Stomakhin snow-plasticity clamp. Matrices are row-major arrays a[3*i+j].
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cfloat>

#define MPM_HD __host__ __device__ __forceinline__

namespace mpm {

// T: particle/grid storage and transfer arithmetic. TS: SVD/polar arithmetic. (CG dot products
// and norms are formed per node in T and added up to FP64 or twice FP32 precision.)
struct PrecFP32  { using T=float;  using TS=float;  static constexpr int id=0; };
struct PrecMixed { using T=float;  using TS=double; static constexpr int id=1; };
struct PrecFP64  { using T=double; using TS=double; static constexpr int id=2; };

template<class T> MPM_HD T mpm_sqrt(T x);
template<> MPM_HD float mpm_sqrt<float>(float x){return sqrtf(x);}
template<> MPM_HD double mpm_sqrt<double>(double x){return sqrt(x);}
template<class T> MPM_HD T mpm_abs(T x){return x<T(0)?-x:x;}
template<class T> MPM_HD T mpm_exp(T x);
template<> MPM_HD float mpm_exp<float>(float x){return expf(x);}
template<> MPM_HD double mpm_exp<double>(double x){return exp(x);}

// ---- 3x3 helpers (row-major) ----
template<class T> MPM_HD void mat_mul(const T* A,const T* B,T* C)          // C = A B
{
#pragma unroll
    for(int i=0;i<3;++i)
#pragma unroll
        for(int j=0;j<3;++j) C[3*i+j]=A[3*i]*B[j]+A[3*i+1]*B[3+j]+A[3*i+2]*B[6+j];
}
template<class T> MPM_HD void mat_mul_bt(const T* A,const T* B,T* C)       // C = A B^T
{
#pragma unroll
    for(int i=0;i<3;++i)
#pragma unroll
        for(int j=0;j<3;++j) C[3*i+j]=A[3*i]*B[3*j]+A[3*i+1]*B[3*j+1]+A[3*i+2]*B[3*j+2];
}
template<class T> MPM_HD void mat_mul_at(const T* A,const T* B,T* C)       // C = A^T B
{
#pragma unroll
    for(int i=0;i<3;++i)
#pragma unroll
        for(int j=0;j<3;++j) C[3*i+j]=A[i]*B[j]+A[3+i]*B[3+j]+A[6+i]*B[6+j];
}
template<class T> MPM_HD T det3(const T* a)
{return a[0]*(a[4]*a[8]-a[5]*a[7])-a[1]*(a[3]*a[8]-a[5]*a[6])+a[2]*(a[3]*a[7]-a[4]*a[6]);}
template<class T> MPM_HD void cofactor3(const T* a,T* C)                   // det(F) F^{-T}
{
    C[0]=a[4]*a[8]-a[5]*a[7]; C[1]=a[5]*a[6]-a[3]*a[8]; C[2]=a[3]*a[7]-a[4]*a[6];
    C[3]=a[2]*a[7]-a[1]*a[8]; C[4]=a[0]*a[8]-a[2]*a[6]; C[5]=a[1]*a[6]-a[0]*a[7];
    C[6]=a[1]*a[5]-a[2]*a[4]; C[7]=a[2]*a[3]-a[0]*a[5]; C[8]=a[0]*a[4]-a[1]*a[3];
}
// d/de cof(F + e dF): product rule on each cofactor entry (reference
// MPM_Constitutive_Model.h:33-46).
template<class T> MPM_HD void cofactor3_diff(const T* a,const T* b,T* C)
{
    C[0]=b[4]*a[8]+a[4]*b[8]-b[5]*a[7]-a[5]*b[7];
    C[1]=b[5]*a[6]+a[5]*b[6]-b[3]*a[8]-a[3]*b[8];
    C[2]=b[3]*a[7]+a[3]*b[7]-b[4]*a[6]-a[4]*b[6];
    C[3]=b[2]*a[7]+a[2]*b[7]-b[1]*a[8]-a[1]*b[8];
    C[4]=b[0]*a[8]+a[0]*b[8]-b[2]*a[6]-a[2]*b[6];
    C[5]=b[1]*a[6]+a[1]*b[6]-b[0]*a[7]-a[0]*b[7];
    C[6]=b[1]*a[5]+a[1]*b[5]-b[2]*a[4]-a[2]*b[4];
    C[7]=b[2]*a[3]+a[2]*b[3]-b[0]*a[5]-a[0]*b[5];
    C[8]=b[0]*a[4]+a[0]*b[4]-b[1]*a[3]-a[1]*b[3];
}

// ---- quadratic B-spline weights (reference MPM_Particle.h:79-100) ----
// x = (X - (center(c) - dx))/dx in [0.5, 1.5); weights of nodes c-1, c, c+1 and their
// derivatives. Products and sums are rounded separately (no contraction) so the weight
// set, and with it the Interior node set, is the same on every machine.
template<class T> MPM_HD void bspline_weights(T x,const T inv_dx,T w[3],T dw[3]);
template<> MPM_HD void bspline_weights<float>(float x,const float inv_dx,float w[3],float dw[3])
{
#ifdef __CUDA_ARCH__
    w[0]=fabsf(__fadd_rn(__fsub_rn(__fmul_rn(__fmul_rn(0.5f,x),x),__fmul_rn(1.5f,x)),1.125f));
    dw[0]=__fmul_rn(__fsub_rn(x,1.5f),inv_dx);
    float y=__fsub_rn(x,1.f);
    w[1]=fabsf(__fadd_rn(-__fmul_rn(y,y),.75f));
    dw[1]=__fmul_rn(__fmul_rn(-2.f,y),inv_dx);
    y=__fsub_rn(y,1.f);
    w[2]=fabsf(__fadd_rn(__fadd_rn(__fmul_rn(__fmul_rn(.5f,y),y),__fmul_rn(1.5f,y)),1.125f));
    dw[2]=__fmul_rn(__fadd_rn(y,1.5f),inv_dx);
#else
    w[0]=fabsf(0.5f*x*x-1.5f*x+1.125f); dw[0]=(x-1.5f)*inv_dx;
    float y=x-1.f; w[1]=fabsf(-y*y+.75f); dw[1]=-2.f*y*inv_dx;
    y-=1.f; w[2]=fabsf(.5f*y*y+1.5f*y+1.125f); dw[2]=(y+1.5f)*inv_dx;
#endif
}
template<> MPM_HD void bspline_weights<double>(double x,const double inv_dx,double w[3],double dw[3])
{
#ifdef __CUDA_ARCH__
    w[0]=fabs(__dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(0.5,x),x),-__dmul_rn(1.5,x)),1.125));
    dw[0]=__dmul_rn(__dadd_rn(x,-1.5),inv_dx);
    double y=__dadd_rn(x,-1.);
    w[1]=fabs(__dadd_rn(-__dmul_rn(y,y),.75));
    dw[1]=__dmul_rn(__dmul_rn(-2.,y),inv_dx);
    y=__dadd_rn(y,-1.);
    w[2]=fabs(__dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(.5,y),y),__dmul_rn(1.5,y)),1.125));
    dw[2]=__dmul_rn(__dadd_rn(y,1.5),inv_dx);
#else
    w[0]=fabs(0.5*x*x-1.5*x+1.125); dw[0]=(x-1.5)*inv_dx;
    double y=x-1.; w[1]=fabs(-y*y+.75); dw[1]=-2.*y*inv_dx;
    y-=1.; w[2]=fabs(.5*y*y+1.5*y+1.125); dw[2]=(y+1.5)*inv_dx;
#endif
}

// ---- 3x3 SVD ----
// F = U diag(s) V^T, U and V rotations, s0 >= s1 >= |s2|, sign of det F on s2 (the
// convention of the Fast_Singular_Value_Decomposition the reference calls,
// MPM_Constitutive_Model.cpp:36). Cyclic Jacobi on the symmetric F^T F (Golub & Van
// Loan, "Matrix Computations", sec. 8.5) with at most `max_sweeps` sweeps, then U from the
// columns of F V by Gram-Schmidt and a cross product.
// With a warm start `V0` (orthonormal columns, e.g. the FP32 solution of the same F) the
// sweeps start from A = V0^T F^T F V0, which is already nearly diagonal. The sweeps stop
// once the off-diagonal mass is below (rel |diag|)^2; rel <= 0 means the epsilon of T.
template<class T,int max_sweeps=6> MPM_HD void svd3(const T* F,T* U,T* s,T* V,const T* V0=nullptr,T rel=T(0))
{
    T v[9]={T(1),T(0),T(0),T(0),T(1),T(0),T(0),T(0),T(1)};
    // A = F^T F, or with a warm start V0^T F^T F V0 = B^T B with B = F V0 (the column dot
    // products of B: 45 multiply-adds instead of 72 through F^T F)
    const T* C=F;
    T B0[9];
    if(V0){
#pragma unroll
        for(int k=0;k<9;++k) v[k]=V0[k];
        mat_mul(F,v,B0);C=B0;}
    T a00=C[0]*C[0]+C[3]*C[3]+C[6]*C[6];
    T a01=C[0]*C[1]+C[3]*C[4]+C[6]*C[7];
    T a02=C[0]*C[2]+C[3]*C[5]+C[6]*C[8];
    T a11=C[1]*C[1]+C[4]*C[4]+C[7]*C[7];
    T a12=C[1]*C[2]+C[4]*C[5]+C[7]*C[8];
    T a22=C[2]*C[2]+C[5]*C[5]+C[8]*C[8];
    const T eps=rel>T(0)?rel:(sizeof(T)==4?T(1.1920929e-7):T(2.220446049250313e-16));
    auto rotate=[&](T& app,T& aqq,T& apq,T& arp,T& arq,int p,int q){
        if(apq==T(0)) return;
        // t = tan of the rotation angle = sgn(theta)/(|theta| + sqrt(theta^2 + 1)) with
        // theta = (aqq - app)/(2 apq). Near the diagonal (warm starts, late sweeps) r =
        // 1/(2 theta) is small and t = 2r/(1 + sqrt(1 + 4r^2)) = r(1 - r^2 + 2r^4) + O(r^7),
        // c = (1 + t^2)^(-1/2) = 1 - t^2/2 + 3t^4/8 + O(t^6): relative errors below 1e-23
        // for |r| <= 1e-4, with one division instead of three divisions and two roots.
        const T d=aqq-app;
        T t,c;
        if(mpm_abs(apq)<=T(1e-4)*mpm_abs(d)){
            const T r=apq/d,r2=r*r;
            t=r*(T(1)-r2+T(2)*r2*r2);
            const T t2=t*t;
            c=T(1)-t2*(T(0.5)-T(0.375)*t2);}
        else{
            const T theta=d/(T(2)*apq);
            t=(theta>=T(0)?T(1):T(-1))/(mpm_abs(theta)+mpm_sqrt(theta*theta+T(1)));
            c=T(1)/mpm_sqrt(t*t+T(1));}
        const T sn=t*c;
        app-=t*apq; aqq+=t*apq; apq=T(0);
        T rp=arp,rq=arq; arp=c*rp-sn*rq; arq=sn*rp+c*rq;    // the remaining off-diagonal pair
#pragma unroll
        for(int k=0;k<3;++k){T vp=v[3*k+p],vq=v[3*k+q];v[3*k+p]=c*vp-sn*vq;v[3*k+q]=sn*vp+c*vq;}
    };
#pragma unroll 1
    for(int sweep=0;sweep<max_sweeps;++sweep){
        // off-diagonal mass below (eps |diag|)^2: further rotations only move rounding noise
        T off=a01*a01+a02*a02+a12*a12,diag=a00*a00+a11*a11+a22*a22;
        if(off<=eps*eps*diag) break;
        rotate(a00,a11,a01,a02,a12,0,1);   // (p,q)=(0,1): the other pair is (a02,a12)
        rotate(a00,a22,a02,a01,a12,0,2);   // (0,2): (a01,a21)
        rotate(a11,a22,a12,a01,a02,1,2);   // (1,2): (a10,a20)
    }
    // sort the eigenvalues of F^T F descending with V's columns
    T e0=a00,e1=a11,e2=a22;
    auto swapc=[&](int i,int j){
#pragma unroll
        for(int k=0;k<3;++k){T t=v[3*k+i];v[3*k+i]=v[3*k+j];v[3*k+j]=t;}};
    if(e1>e0){T t=e0;e0=e1;e1=t;swapc(0,1);}
    if(e2>e0){T t=e0;e0=e2;e2=t;swapc(0,2);}
    if(e2>e1){T t=e1;e1=e2;e2=t;swapc(1,2);}
    if(det3(v)<T(0)){v[2]=-v[2];v[5]=-v[5];v[8]=-v[8];}
    T B[9];mat_mul(F,v,B);
    T b0[3]={B[0],B[3],B[6]},b1[3]={B[1],B[4],B[7]},b2[3]={B[2],B[5],B[8]};
    const T tiny=sizeof(T)==4?T(1e-30):T(1e-290);
    T n0=mpm_sqrt(b0[0]*b0[0]+b0[1]*b0[1]+b0[2]*b0[2]);
    T u0[3]={T(1),T(0),T(0)};
    if(n0>tiny){T r=T(1)/n0;u0[0]=b0[0]*r;u0[1]=b0[1]*r;u0[2]=b0[2]*r;}
    T p=u0[0]*b1[0]+u0[1]*b1[1]+u0[2]*b1[2];
    T u1[3]={b1[0]-p*u0[0],b1[1]-p*u0[1],b1[2]-p*u0[2]};
    T n1=mpm_sqrt(u1[0]*u1[0]+u1[1]*u1[1]+u1[2]*u1[2]);
    if(n1>tiny*T(100)*(n0>T(1)?n0:T(1))){T r=T(1)/n1;u1[0]*=r;u1[1]*=r;u1[2]*=r;}
    else{ // any unit vector orthogonal to u0
        int m=0;if(mpm_abs(u0[1])<mpm_abs(u0[m])) m=1;if(mpm_abs(u0[2])<mpm_abs(u0[m])) m=2;
        T e[3]={T(0),T(0),T(0)};e[m]=T(1);T q=u0[m];
        u1[0]=e[0]-q*u0[0];u1[1]=e[1]-q*u0[1];u1[2]=e[2]-q*u0[2];
        T r=T(1)/mpm_sqrt(u1[0]*u1[0]+u1[1]*u1[1]+u1[2]*u1[2]);u1[0]*=r;u1[1]*=r;u1[2]*=r;}
    T u2[3]={u0[1]*u1[2]-u0[2]*u1[1],u0[2]*u1[0]-u0[0]*u1[2],u0[0]*u1[1]-u0[1]*u1[0]};
#pragma unroll
    for(int k=0;k<3;++k){U[3*k]=u0[k];U[3*k+1]=u1[k];U[3*k+2]=u2[k];}
    s[0]=u0[0]*b0[0]+u0[1]*b0[1]+u0[2]*b0[2];
    s[1]=u1[0]*b1[0]+u1[1]*b1[1]+u1[2]*b1[2];
    s[2]=u2[0]*b2[0]+u2[1]*b2[1]+u2[2]*b2[2];
#pragma unroll
    for(int k=0;k<9;++k) V[k]=v[k];
}

// ---- constitutive model (reference MPM_Constitutive_Model.cpp:32-76) ----
// 1/sqrt(x) for x within 1e-4 of 1: 1 - e/2 + 3e^2/8 - 5e^3/16 with e = x - 1 (next term
// 35e^4/128, below 3e-17); otherwise the root and the division.
template<class T> MPM_HD T rsqrt_near1(T x)
{
    const T e=x-T(1);
    if(mpm_abs(e)<=T(1e-4)) return T(1)-e*(T(0.5)-e*(T(0.375)-T(0.3125)*e));
    return T(1)/mpm_sqrt(x);
}
// Columns of V made orthonormal in T (Gram-Schmidt, then a cross product for the third).
// Columns that are already unit length to ~1e-7 (an FP32 solution) take the series for
// the inverse norms.
template<class T> MPM_HD void orthonormalize3(T* v)
{
    T n=rsqrt_near1(v[0]*v[0]+v[3]*v[3]+v[6]*v[6]);
    v[0]*=n;v[3]*=n;v[6]*=n;
    const T p=v[0]*v[1]+v[3]*v[4]+v[6]*v[7];
    v[1]-=p*v[0];v[4]-=p*v[3];v[7]-=p*v[6];
    n=rsqrt_near1(v[1]*v[1]+v[4]*v[4]+v[7]*v[7]);
    v[1]*=n;v[4]*=n;v[7]*=n;
    v[2]=v[3]*v[7]-v[6]*v[4];v[5]=v[6]*v[1]-v[0]*v[7];v[8]=v[0]*v[4]-v[3]*v[1];
}

// Refines an approximate polar rotation R of F (R close to the exact factor R*, F = R* S*
// with S* symmetric): the skew correction W with W S + S W = S - S^T (S = R^T F) is the
// first-order rotation error (the same 3x3 system as dR, reference
// MPM_Constitutive_Model.h:56-69); R <- R (I + W), then (if `bjorck`) one Bjorck step
// R <- R (3I - R^T R)/2 restores orthonormality. Each pass squares the error, so from an
// FP32 start one pass without the Bjorck step leaves an O(1e-14) error, far below the FP32
// rounding of the stored result.
template<class T> MPM_HD T recip(T x);
template<> MPM_HD float recip<float>(float x){return 1.f/x;}
template<> MPM_HD double recip<double>(double x)
{   // FP32 seed and two Newton steps: each step squares the relative error (1e-7 -> 1e-14
    // -> below FP64 rounding), so the result is 1/x to FP64 rounding error. The FP32 seed
    // needs |x| inside the FP32 normal range; outside it (never for the O(1) determinants
    // the polar refinement passes) the plain FP64 division is used.
    const double ax=x<0.?-x:x;
    if(!(ax>=1e-37&&ax<=1e37)) return 1.0/x;
#ifdef __CUDA_ARCH__
    double y=(double)__frcp_rn((float)x);
#else
    double y=(double)(1.f/(float)x);
#endif
    y=y*(2.0-x*y);y=y*(2.0-x*y);
    return y;
}
template<class T> MPM_HD void polar_refine3(const T* F,T* R,bool bjorck=true)
{
    T S[9];mat_mul_at(R,F,S);
    const T s01=T(0.5)*(S[1]+S[3]),s02=T(0.5)*(S[2]+S[6]),s12=T(0.5)*(S[5]+S[7]);
    const T k00=S[4]+S[0],k01=s12,k02=-s02,k11=S[8]+S[0],k12=s01,k22=S[8]+S[4];
    const T L0=S[3]-S[1],L1=S[6]-S[2],L2=S[7]-S[5];
    const T c00=k11*k22-k12*k12,c01=k02*k12-k01*k22,c02=k01*k12-k02*k11;
    const T c11=k00*k22-k02*k02,c12=k01*k02-k00*k12,c22=k00*k11-k01*k01;
    const T inv=recip<T>(k00*c00+k01*c01+k02*c02);
    const T a=(c00*L0+c01*L1+c02*L2)*inv,b=(c01*L0+c11*L1+c12*L2)*inv,c=(c02*L0+c12*L1+c22*L2)*inv;
    T Rn[9];
#pragma unroll
    for(int i=0;i<3;++i){
        const T r0=R[3*i],r1=R[3*i+1],r2=R[3*i+2];
        Rn[3*i]=r0+r1*a+r2*b;Rn[3*i+1]=r1-r0*a+r2*c;Rn[3*i+2]=r2-r0*b-r1*c;}
    if(!bjorck){
#pragma unroll
        for(int k=0;k<9;++k) R[k]=Rn[k];
        return;}
    T G[9];mat_mul_at(Rn,Rn,G);
#pragma unroll
    for(int k=0;k<9;++k) G[k]=(k%4==0?T(1.5):T(0))-T(0.5)*G[k];
    mat_mul(Rn,G,R);
}

// Sum of the six products sum_k (a_k b_k - c_k d_k) over k = 0..2, evaluated as if in twice
// FP32 precision and then rounded: Dot2 (Ogita, Rump & Oishi, "Accurate sum and dot
// product", SIAM J. Sci. Comput. 26, 2005). Each product is split exactly into p + e with
// one fused multiply-add (e = fma(a, b, -p)), the p's are summed with Knuth's error-free
// TwoSum and all error terms are added at the end. The error is below
// 2^-24 |result| + (6 * 2^-24)^2 sum |terms|.
MPM_HD float dot2_skew3(const float* a,const float* b,const float* c,const float* d,int sa,int sb)
{
    float s=0.f,err=0.f;
#pragma unroll
    for(int k=0;k<6;++k){
        const int i=k>>1;
        const float x=(k&1)?-c[sa*i]:a[sa*i],y=(k&1)?d[sb*i]:b[sb*i];
        const float p=x*y,e=fmaf(x,y,-p);              // x y = p + e exactly
        const float t=s+p,z=t-s,q=(s-(t-z))+(p-z);     // s + p = t + q exactly (TwoSum)
        s=t;err+=q+e;}
    return s+err;
}

// det F of an FP32 matrix as the FP64 determinant would round it: the six triple products
// a_i a_j a_k each split into an exact product pair of a_i a_j (one FMA) times a_k (again
// split exactly; the pair's low part times a_k adds an error below 2^-48), summed with
// TwoSum and the error terms added at the end (Dot2). Used by the mixed variant, where the
// FP64 pipe runs at 1/64 of the FP32 rate.
MPM_HD float det3_dot2(const float* a)
{
    const int idx[6][3]={{0,4,8},{1,5,6},{2,3,7},{2,4,6},{0,5,7},{1,3,8}};
    float s=0.f,err=0.f;
#pragma unroll
    for(int t=0;t<6;++t){
        const float x=a[idx[t][0]],y=a[idx[t][1]],z=a[idx[t][2]];
        const float p=x*y,e=fmaf(x,y,-p);               // x y = p + e exactly
        float q=p*z;const float eq=fmaf(p,z,-q);        // p z = q + eq exactly
        float r=fmaf(e,z,eq);                            // the small parts of x y z
        if(t>=3){q=-q;r=-r;}
        const float u=s+q,zz=u-s,c=(s-(u-zz))+(q-zz);    // TwoSum
        s=u;err+=c+r;}
    return s+err;
}

// Mixed-precision form of one polar_refine3 pass without the Bjorck step, for FP32 F and an
// FP32 rotation R. The correction W is ~1e-7, so only its source needs more than FP32: the
// skew part L of R^T F, a difference of nearly equal sums. L is evaluated to twice FP32
// precision by dot2_skew3 (products split exactly, sums compensated), which gives the
// same rounded L as an FP64 evaluation (where the FP32 products are exact) without any
// FP64 operation: on GB300 the FP64 rate is 1/64 of FP32, and the FP64 form cost about a
// fifth of the whole P2G on the 64-scene batch. The symmetric 3x3 system for W and the
// update R + R W stay in FP32: their relative errors (~1e-7) scale W, i.e. ~1e-14
// absolute, far below the FP32 rounding of the stored rotation.
MPM_HD void polar_refine_mixed(const float* F,float* R)
{
    float S[9];mat_mul_at(R,F,S);
    const float s01=0.5f*(S[1]+S[3]),s02=0.5f*(S[2]+S[6]),s12=0.5f*(S[5]+S[7]);
    const float k00=S[4]+S[0],k01=s12,k02=-s02,k11=S[8]+S[0],k12=s01,k22=S[8]+S[4];
    // L0 = sum_k R[k][1] F[k][0] - R[k][0] F[k][1], L1 = (2,0)-(0,2), L2 = (2,1)-(1,2)
    const float l0=dot2_skew3(R+1,F,R,F+1,3,3),l1=dot2_skew3(R+2,F,R,F+2,3,3),l2=dot2_skew3(R+2,F+1,R+1,F+2,3,3);
    const float c00=k11*k22-k12*k12,c01=k02*k12-k01*k22,c02=k01*k12-k02*k11;
    const float c11=k00*k22-k02*k02,c12=k01*k02-k00*k12,c22=k00*k11-k01*k01;
    const float inv=1.f/(k00*c00+k01*c01+k02*c02);
    const float a=(c00*l0+c01*l1+c02*l2)*inv,b=(c01*l0+c11*l1+c12*l2)*inv,c=(c02*l0+c12*l1+c22*l2)*inv;
    float Rn[9];
#pragma unroll
    for(int i=0;i<3;++i){
        const float r0=R[3*i],r1=R[3*i+1],r2=R[3*i+2];
        Rn[3*i]=r0+(r1*a+r2*b);Rn[3*i+1]=r1+(r2*c-r0*a);Rn[3*i+2]=r2-(r0*b+r1*c);}
#pragma unroll
    for(int k=0;k<9;++k) R[k]=Rn[k];
}

// ---- FP32 pairs ----
// An unevaluated sum h + l of two FP32 numbers. Products and sums that the error terms depend
// on are rounded one by one (never contracted into a fused multiply-add).
struct F2x { float h,l; };
MPM_HD float ff_mul(float a,float b)
{
#ifdef __CUDA_ARCH__
    return __fmul_rn(a,b);
#else
    return a*b;
#endif
}
MPM_HD float ff_add(float a,float b)
{
#ifdef __CUDA_ARCH__
    return __fadd_rn(a,b);
#else
    return a+b;
#endif
}
// a0 b0 + a1 b1 + a2 b2 + c: the products split exactly by one FMA each, their sum by TwoSum,
// the error terms and c (small) added up in l (Dot2, as in dot2_skew3). h + l has an error
// below 2^-44 sum |terms|.
MPM_HD F2x ff_dot3(float a0,float b0,float a1,float b1,float a2,float b2,float c=0.f)
{
    const float p0=ff_mul(a0,b0),p1=ff_mul(a1,b1),p2=ff_mul(a2,b2);
    const float s=ff_add(p0,p1),z=ff_add(s,-p0),q=ff_add(ff_add(p0,-ff_add(s,-z)),ff_add(p1,-z));
    const float t=ff_add(s,p2),y=ff_add(t,-s),r=ff_add(ff_add(s,-ff_add(t,-y)),ff_add(p2,-y));
    return F2x{t,(fmaf(a0,b0,-p0)+fmaf(a1,b1,-p1))+(fmaf(a2,b2,-p2)+c)+(q+r)};
}
MPM_HD F2x ff_norm(F2x a){const float h=ff_add(a.h,a.l);return F2x{h,ff_add(a.l,-ff_add(h,-a.h))};}
MPM_HD F2x ff_prod(F2x a,F2x b){const float p=ff_mul(a.h,b.h);return ff_norm(F2x{p,fmaf(a.h,b.h,-p)+(a.h*b.l+a.l*b.h)});}

// The clamped plasticity update of the mixed variant from the FP32 SVD F ~ U diag(s) V^T
// (s2 well above 0), to FP32 rounding of the exact result, without FP64 operations: the FP64
// pipe runs at 1/64 of the FP32 rate, and the FP64 Jacobi this replaces took four fifths
// of P2G once most particles yield (1.94M particles, 81 % clamped: P2G 1.79 -> 0.65 ms).
// One step of first-order correction, its inputs evaluated to twice FP32 precision:
//   dU = U^T U - I, dV = V^T V - I   (the orthonormal factors are U (I - dU/2), V (I - dV/2)),
//   M = U^T F V - (dU D + D dV)/2 = D + E with D diagonal and E ~ 1e-7.
// A function f of the singular values changes along E by the divided differences of f (Daleckii
// and Krein; for singular values, Noferini, "A formula for the Frechet derivative of a
// generalized matrix function", SIAM J. Matrix Anal. Appl. 38, 2017):
//   N_ij = (f_i - f_j)/(d_i - d_j) (E_ij + E_ji)/2 + (f_i + f_j)/(d_i + d_j) (E_ij - E_ji)/2,
// bounded for the clamp (its first quotient lies in [0, 1]); f = 1 gives the rotation. The
// neglected terms are of order E^2. Fe, Re = U (f + N - (dU f + f dV)/2) V^T, the leading
// product to twice FP32 precision.
//
// For bands wider than CLAMP_MIN_BAND: only then are no singular values near both limits (below,
// within 1e-4), and limits that cross (where the lower one wins) are left to the plain form.
constexpr float CLAMP_MIN_BAND=3e-4f;
MPM_HD void clamp_refined(float* Fe,float& Jp,const float* U,const float* V,const float cy,const float sy,float* Re,float& Je)
{
    float dU[9],dV[9];               // symmetric
#pragma unroll
    for(int i=0;i<3;++i)
#pragma unroll
        for(int j=i;j<3;++j){
            const F2x u=ff_dot3(U[i],U[j],U[3+i],U[3+j],U[6+i],U[6+j]),v=ff_dot3(V[i],V[j],V[3+i],V[3+j],V[6+i],V[6+j]);
            dU[3*i+j]=dU[3*j+i]=(i==j?u.h-1.f:u.h)+u.l;
            dV[3*i+j]=dV[3*j+i]=(i==j?v.h-1.f:v.h)+v.l;}
    F2x D[3];float E[9];
#pragma unroll
    for(int j=0;j<3;++j){
        F2x t[3];                     // column j of F V
#pragma unroll
        for(int k=0;k<3;++k) t[k]=ff_dot3(Fe[3*k],V[j],Fe[3*k+1],V[3+j],Fe[3*k+2],V[6+j]);
#pragma unroll
        for(int i=0;i<3;++i){
            const F2x m=ff_dot3(U[i],t[0].h,U[3+i],t[1].h,U[6+i],t[2].h,U[i]*t[0].l+U[3+i]*t[1].l+U[6+i]*t[2].l);
            if(i==j) D[i]=m; else E[3*i+j]=m.h+m.l;}}
#pragma unroll
    for(int i=0;i<3;++i){D[i].l-=0.5f*D[i].h*(dU[4*i]+dV[4*i]);D[i]=ff_norm(D[i]);}
    // e[i][j] of the sum above, of which the symmetric part S enters with f's quotient
    float S01,S02,S12,w01,w02,w12;
    auto split=[&](int i,int j,float& sym,float& w){
        const float di=D[i].h,dj=D[j].h,u=0.5f*dU[3*i+j],v=0.5f*dV[3*i+j];
        const float e1=E[3*i+j]-(u*dj+di*v),e2=E[3*j+i]-(u*di+dj*v);
        sym=0.5f*(e1+e2);w=(e1-e2)/(di+dj);};
    split(0,1,S01,w01);split(0,2,S02,w02);split(1,2,S12,w12);
    // The first order is not enough where singular values lie on both sides of one limit and
    // about E or less apart. Those within 1e-4 of a limit (where E^2 over the gap is far below
    // the rounding) have their small block, D - limit and S, diagonalised: Q, lam.
    F2x f[3],q=F2x{1.f,0.f},jf=F2x{1.f,0.f};
    const float rlo=0.f-cy,rhi=0.f-sy;
    auto off=[&](int i,float r){return ff_add(D[i].h,r)+D[i].l;};
    auto count=[&](float r){return (mpm_abs(off(0,r))<1e-4f)+(mpm_abs(off(1,r))<1e-4f)+(mpm_abs(off(2,r))<1e-4f);};
    const float k=count(rlo)>=2?cy:count(rhi)>=2?sy:0.f;
    bool near[3]={false,false,false};
    float P01=0.f,P02=0.f,P12=0.f;
    if(k!=0.f){
        float a[3];
#pragma unroll
        for(int i=0;i<3;++i){a[i]=off(i,-k);near[i]=mpm_abs(a[i])<1e-4f;}
        float a01=near[0]&&near[1]?S01:0.f,a02=near[0]&&near[2]?S02:0.f,a12=near[1]&&near[2]?S12:0.f;
        float Q[9]={1.f,0.f,0.f,0.f,1.f,0.f,0.f,0.f,1.f};
        auto rotate=[&](float& app,float& aqq,float& apq,float& arp,float& arq,int p,int r){
            if(apq==0.f) return;
            const float th=(aqq-app)/(2.f*apq);
            const float t=(th>=0.f?1.f:-1.f)/(mpm_abs(th)+mpm_sqrt(th*th+1.f)),c=1.f/mpm_sqrt(t*t+1.f),sn=t*c;
            app-=t*apq;aqq+=t*apq;apq=0.f;
            const float rp=arp,rq=arq;arp=c*rp-sn*rq;arq=sn*rp+c*rq;
#pragma unroll
            for(int m=0;m<3;++m){const float vp=Q[3*m+p],vq=Q[3*m+r];Q[3*m+p]=c*vp-sn*vq;Q[3*m+r]=sn*vp+c*vq;}};
#pragma unroll 1
        for(int sweep=0;sweep<3;++sweep){
            rotate(a[0],a[1],a01,a02,a12,0,1);rotate(a[0],a[2],a02,a01,a12,0,2);rotate(a[1],a[2],a12,a01,a02,1,2);}
        float ph[3];
#pragma unroll
        for(int m=0;m<3;++m){
            ph[m]=near[m]?fminf(fmaxf(a[m],cy-k),sy-k):0.f;        // f(k + lam) - k
            if(near[m]){q=ff_prod(q,F2x{1.f,(a[m]-ph[m])/(k+ph[m])});jf=ff_prod(jf,F2x{k,ph[m]});}}
        auto back=[&](int i,int j){return Q[3*i]*ph[0]*Q[3*j]+Q[3*i+1]*ph[1]*Q[3*j+1]+Q[3*i+2]*ph[2]*Q[3*j+2];};
        P01=back(0,1);P02=back(0,2);P12=back(1,2);
#pragma unroll
        for(int i=0;i<3;++i) if(near[i]) f[i]=F2x{k,back(i,i)};}
#pragma unroll
    for(int i=0;i<3;++i) if(!near[i]){
        // the sign of D - limit decides, as one rounding of the exact value would
        const bool up=off(i,rhi)>0.f,lo=off(i,rlo)<0.f;
        f[i]=up?F2x{sy,0.f}:lo?F2x{cy,0.f}:D[i];
        jf=ff_prod(jf,f[i]);
        if(up||lo){                  // q *= D / f
            const float r=1.f/f[i].h,qh=D[i].h*r;
            q=ff_prod(q,F2x{qh,(fmaf(-qh,f[i].h,D[i].h)+D[i].l)*r});}}
    const float jh=ff_mul(Jp,q.h);
    Jp=jh+(fmaf(Jp,q.h,-jh)+Jp*q.l);
    Je=jf.h+jf.l;
    float C[9],W[9];                 // corrections of Fe and of Re inside U (.) V^T
#pragma unroll
    for(int i=0;i<3;++i){
        C[4*i]=f[i].l-0.5f*f[i].h*(dU[4*i]+dV[4*i]);
        W[4*i]=-0.5f*(dU[4*i]+dV[4*i]);}
    auto couple=[&](int i,int j,float sym,float w,float P){
        const float fi=f[i].h+f[i].l,fj=f[j].h+f[j].l,u=0.5f*dU[3*i+j],v=0.5f*dV[3*i+j];
        const float gap=ff_add(D[i].h,-D[j].h)+(D[i].l-D[j].l),num=ff_add(f[i].h,-f[j].h)+(f[i].l-f[j].l);
        // equal singular values: the clamp's slope there (0 beyond a limit, else 1)
        const float a=gap!=0.f?fminf(fmaxf(num/gap,0.f),1.f):(fi==sy||fi==cy?0.f:1.f);
        const float sm=near[i]&&near[j]?P:a*sym,sk=0.5f*(fi+fj)*w;
        C[3*i+j]=sm+sk-(u*fj+fi*v);C[3*j+i]=sm-sk-(u*fi+fj*v);
        W[3*i+j]=w-(u+v);W[3*j+i]=-w-(u+v);};
    couple(0,1,S01,w01,P01);couple(0,2,S02,w02,P02);couple(1,2,S12,w12,P12);
#pragma unroll
    for(int i=0;i<3;++i){
        float ph[3],pl[3],cf[3],cr[3];      // row i of U f (split exactly), U C, U W
#pragma unroll
        for(int k=0;k<3;++k){
            ph[k]=ff_mul(U[3*i+k],f[k].h);pl[k]=fmaf(U[3*i+k],f[k].h,-ph[k]);
            cf[k]=U[3*i]*C[k]+U[3*i+1]*C[3+k]+U[3*i+2]*C[6+k];
            cr[k]=U[3*i]*W[k]+U[3*i+1]*W[3+k]+U[3*i+2]*W[6+k];}
#pragma unroll
        for(int j=0;j<3;++j){
            const float v0=V[3*j],v1=V[3*j+1],v2=V[3*j+2];
            const F2x x=ff_dot3(ph[0],v0,ph[1],v1,ph[2],v2,(pl[0]+cf[0])*v0+(pl[1]+cf[1])*v1+(pl[2]+cf[2])*v2);
            Fe[3*i+j]=x.h+x.l;
            const F2x y=ff_dot3(U[3*i],v0,U[3*i+1],v1,U[3*i+2],v2,cr[0]*v0+cr[1]*v1+cr[2]*v2);
            Re[3*i+j]=y.h+y.l;}}
}

// The clamp by the FP64 Jacobi SVD (to `rel`, see svd3) warm-started from the FP32 V.
template<class T> MPM_HD void clamp_fp64(T* Fe,T& Jp,const float* V32,const int plastic,const T cy,const T sy,const double rel,T* Re,T& Je)
{
    double F[9],U[9],s[3],V[9],V0[9];
#pragma unroll
    for(int k=0;k<9;++k){F[k]=(double)Fe[k];V0[k]=(double)V32[k];}
    orthonormalize3(V0);
    svd3<double,4>(F,U,s,V,V0,rel);
    const double prod_s=s[0]*s[1]*s[2];
    if(plastic){
#pragma unroll
        for(int i=0;i<3;++i){if(s[i]>(double)sy) s[i]=(double)sy;if(s[i]<(double)cy) s[i]=(double)cy;}
        Jp=(T)((double)Jp*(prod_s/(s[0]*s[1]*s[2])));
#pragma unroll
        for(int i=0;i<3;++i)
#pragma unroll
            for(int j=0;j<3;++j) Fe[3*i+j]=(T)(U[3*i]*s[0]*V[3*j]+U[3*i+1]*s[1]*V[3*j+1]+U[3*i+2]*s[2]*V[3*j+2]);}
    Je=(T)(s[0]*s[1]*s[2]);
    double R[9];mat_mul_bt(U,V,R);
#pragma unroll
    for(int k=0;k<9;++k) Re[k]=(T)R[k];
}
// The same out of line, for the mixed variant, where it is rare: inlined, its code would push
// P2G's loop out of the instruction cache. An FP64 SVD to 1e-12 relative (one sweep from
// the FP32 start, as a rule) is four orders below the FP32 rounding of Fe, Jp and Re.
struct ClampArgs { float Fe[9],V32[9],Jp,cy,sy; };
struct ClampResult { float Fe[9],Re[9],Jp,Je; };
static __host__ __device__ __noinline__ ClampResult clamp_fp64_cold(ClampArgs a)
{
    ClampResult r;r.Jp=a.Jp;
    for(int k=0;k<9;++k) r.Fe[k]=a.Fe[k];
    clamp_fp64<float>(r.Fe,r.Jp,a.V32,1,a.cy,a.sy,1e-12,r.Re,r.Je);
    return r;
}

// Polar rotation of F near a rotation, without an SVD: with e = F^T F - I,
//   R = F (I + e)^(-1/2) = F + F e (-1/2 + e (3/8 - e (5/16 - e 35/128))) + O(63/256 |e|^5).
// e is evaluated to twice FP32 precision and the correction added last, so that R is the exact
// rotation rounded to FP32, but for the series' end: below 2e-10 for |e| <= 0.0149 (Frobenius
// norm, a bound of the eigenvalues of F^T F). Returns false, R untouched, when |e|^2 >= lim2
// or det F < 0: e is as small near a reflection, whose least singular value is negative and
// whose polar rotation is not F (1 + e)^(-1/2).
constexpr float POLAR_SERIES_MAX=0.0149f;
MPM_HD bool polar_near(const float* F,float lim2,float* R)
{
    float c[6];                      // e from plain FP32 products, for the test: 00, 01, 02, 11, 12, 22
    c[0]=F[0]*F[0]+F[3]*F[3]+(F[6]*F[6]-1.f);c[1]=F[0]*F[1]+F[3]*F[4]+F[6]*F[7];c[2]=F[0]*F[2]+F[3]*F[5]+F[6]*F[8];
    c[3]=F[1]*F[1]+F[4]*F[4]+(F[7]*F[7]-1.f);c[4]=F[1]*F[2]+F[4]*F[5]+F[7]*F[8];c[5]=F[2]*F[2]+F[5]*F[5]+(F[8]*F[8]-1.f);
    if(!(c[0]*c[0]+c[3]*c[3]+c[5]*c[5]+2.f*(c[1]*c[1]+c[2]*c[2]+c[4]*c[4])<lim2)) return false;
    if(!(det3(F)>0.f)) return false;          // here |det F| is within 3 % of 1
    float e[6];
    {   const int a[6]={0,0,0,1,1,2},b[6]={0,1,2,1,2,2};
#pragma unroll
        for(int k=0;k<6;++k){
            const F2x d=ff_dot3(F[a[k]],F[b[k]],F[3+a[k]],F[3+b[k]],F[6+a[k]],F[6+b[k]]);
            e[k]=(a[k]==b[k]?d.h-1.f:d.h)+d.l;}}
    // H <- s I + e H, symmetric (polynomials of e commute)
    float H[6];
#pragma unroll
    for(int k=0;k<6;++k) H[k]=e[k]*0.2734375f;
    auto horner=[&](float s){
        const float h0=H[0]+s,h1=H[1],h2=H[2],h3=H[3]+s,h4=H[4],h5=H[5]+s;
        H[0]=e[0]*h0+e[1]*h1+e[2]*h2;H[1]=e[0]*h1+e[1]*h3+e[2]*h4;H[2]=e[0]*h2+e[1]*h4+e[2]*h5;
        H[3]=e[1]*h1+e[3]*h3+e[4]*h4;H[4]=e[1]*h2+e[3]*h4+e[4]*h5;H[5]=e[2]*h2+e[4]*h4+e[5]*h5;};
    horner(-0.3125f);horner(0.375f);horner(-0.5f);
#pragma unroll
    for(int i=0;i<3;++i){
        const float f0=F[3*i],f1=F[3*i+1],f2=F[3*i+2];
        R[3*i]=f0+(f0*H[0]+f1*H[1]+f2*H[2]);R[3*i+1]=f1+(f0*H[1]+f1*H[3]+f2*H[4]);R[3*i+2]=f2+(f0*H[2]+f1*H[4]+f2*H[5]);}
    return true;
}

// Hardened Lame parameters (reference :53-60).
template<class T> MPM_HD void harden(const T Jp,const T lambda0,const T mu0,const int plastic,const T hardening,const T hardening_max,T& lambda,T& mu)
{
    if(plastic){
        T power=hardening*(T(1)-Jp);if(power>hardening_max) power=hardening_max;
        const T e=mpm_exp<T>(power);
        lambda=e*lambda0;mu=e*mu0;}
    else{lambda=lambda0;mu=mu0;}
}
// Precompute: SVD of Fe, clamp of the singular values to [cy, sy], Jp update (det of the
// reference's Fp <- V S^-1 U^T Fe Fp), Fe <- U S_hat V^T, hardened Lame parameters,
// Re = U V^T. Writes Fe, Jp in place (rounded to T).
//
// FP32 storage: a Fe near a rotation and for certain inside the yield band takes polar_near.
// TS == float: everything in FP32. TS == double (mixed and FP64 variants): the SVD is
// first done in FP32. If those singular values lie inside [cy, sy] by a margin far above
// the FP32 error, no clamp happens in exact arithmetic, so Fe and Jp are unchanged and
// only the polar rotation Re is needed, refined in FP64 from the FP32 U V^T by
// polar_refine3 or polar_refine_mixed. Otherwise the mixed variant corrects the FP32 SVD to
// FP32 rounding of the exact clamp (clamp_refined); for singular values far from 1, where the
// correction's quotients are not well conditioned, for a yield band that is hardly one
// (CLAMP_MIN_BAND) and in the FP64 variant the FP64 Jacobi SVD runs, warm-started from the
// FP32 V, and clamp and reconstruction are done in FP64.
template<class T,class TS> MPM_HD void precompute(T* Fe,T& Jp,const T lambda0,const T mu0,
    const int plastic,const T hardening,const T cy,const T sy,const T hardening_max,
    T* Re,T& lambda,T& mu,T& Je)
{
    float F32[9],U32[9],s32[3],V32[9];
#pragma unroll
    for(int k=0;k<9;++k) F32[k]=(float)Fe[k];
    const float margin=1e-5f;
    if constexpr(sizeof(T)==4){
        // no clamp for certain, all singular values inside the yield band: only the rotation is
        // needed (unstrained and lightly strained bodies; the SVD below took half of P2G there)
        const float top=fmaxf(sy-margin,0.f);       // a limit below -1 has a square above 1, too
        const float lim=plastic?fminf(fminf(top*top-1.f,1.f-(cy+margin)*(cy+margin)),POLAR_SERIES_MAX):POLAR_SERIES_MAX;
        if(lim>0.f&&polar_near(F32,lim*lim,Re)){
            Je=det3_dot2(F32);
            harden(Jp,lambda0,mu0,plastic,hardening,hardening_max,lambda,mu);
            return;}}
    svd3<float>(F32,U32,s32,V32);
    const bool inside=s32[0]<(float)sy-margin&&s32[2]>(float)cy+margin;
    if constexpr(sizeof(TS)==4){
        if(plastic){
            const T prod_s=s32[0]*s32[1]*s32[2];
#pragma unroll
            for(int i=0;i<3;++i){if(s32[i]>sy) s32[i]=sy;if(s32[i]<cy) s32[i]=cy;}
            const T prod_hat=s32[0]*s32[1]*s32[2];
            Jp=Jp*(prod_s/prod_hat);
#pragma unroll
            for(int i=0;i<3;++i)
#pragma unroll
                for(int j=0;j<3;++j) Fe[3*i+j]=U32[3*i]*s32[0]*V32[3*j]+U32[3*i+1]*s32[1]*V32[3*j+1]+U32[3*i+2]*s32[2]*V32[3*j+2];}
        Je=s32[0]*s32[1]*s32[2];
        mat_mul_bt(U32,V32,Re);}
    else if(plastic&&!inside){
        if constexpr(sizeof(T)==8) clamp_fp64<T>(Fe,Jp,V32,plastic,cy,sy,0.,Re,Je);
        else if(s32[2]>0.25f&&s32[0]<4.f&&sy-cy>CLAMP_MIN_BAND) clamp_refined(Fe,Jp,U32,V32,cy,sy,Re,Je);
        else{
            ClampArgs a;a.Jp=Jp;a.cy=cy;a.sy=sy;
#pragma unroll
            for(int k=0;k<9;++k){a.Fe[k]=Fe[k];a.V32[k]=V32[k];}
            const ClampResult r=clamp_fp64_cold(a);
#pragma unroll
            for(int k=0;k<9;++k){Fe[k]=r.Fe[k];Re[k]=r.Re[k];}
            Jp=r.Jp;Je=r.Je;}}
    else{
        float R32[9];mat_mul_bt(U32,V32,R32);
        if constexpr(sizeof(T)==8){
            // FP64 variant: to FP64 accuracy
            TS F[9],R[9];
#pragma unroll
            for(int k=0;k<9;++k){F[k]=(TS)Fe[k];R[k]=(TS)R32[k];}
            polar_refine3(F,R);polar_refine3(F,R);
#pragma unroll
            for(int k=0;k<9;++k) Re[k]=(T)R[k];
            Je=(T)det3(F);}
        else{
            // mixed (FP32 Fe and Re): the rounding-sensitive skew residual and det Fe to
            // twice FP32 precision (what FP64 evaluation rounds to), without FP64 operations
            polar_refine_mixed(F32,R32);
#pragma unroll
            for(int k=0;k<9;++k) Re[k]=(T)R32[k];
            Je=(T)det3_dot2(F32);}}
    harden(Jp,lambda0,mu0,plastic,hardening,hardening_max,lambda,mu);
}

// The stress and its differential as the reference writes them: for the host checks, which hold
// them to the oracle; the kernels use the form of HessianData below.
// First Piola-Kirchhoff stress P = 2 mu (Fe - Re) + lambda (Je-1) cof(Fe), reference :63-67.
template<class T> MPM_HD void stress_P(const T* Fe,const T* Re,const T lambda,const T mu,const T Je,T* P)
{
    T H[9];cofactor3(Fe,H);
    const T c=lambda*(Je-T(1)),m2=T(2)*mu;
#pragma unroll
    for(int k=0;k<9;++k) P[k]=m2*(Fe[k]-Re[k])+c*H[k];
}

// Differential of P along dF, reference :71-76 with dR from MPM_Constitutive_Model.h:56-69:
// dP = 2 mu (dF - dR) + lambda (H:dF) H + lambda (Je-1) dH, with R^T dR the skew matrix W
// solving W S + S W = M - M^T (M = R^T dF, S = R^T Fe), a 3x3 system solved by the adjugate.
// Je and H are recomputed from Fe (Je = det Fe, H = cof Fe).
template<class T> MPM_HD void dP_dF(const T* Fe,const T* Re,const T lambda,const T mu,const T* dF,T* dP)
{
    T H[9];cofactor3(Fe,H);
    const T Je=det3(Fe);
    T M[9],S[9];mat_mul_at(Re,dF,M);mat_mul_at(Re,Fe,S);
    const T k00=S[4]+S[0],k01=S[7],k02=-S[6];
    const T k11=S[8]+S[0],k12=S[3];
    const T k22=S[8]+S[4];
    const T L0=M[3]-M[1],L1=M[6]-M[2],L2=M[7]-M[5];
    // symmetric K: adjugate
    const T c00=k11*k22-k12*k12,c01=k02*k12-k01*k22,c02=k01*k12-k02*k11;
    const T c11=k00*k22-k02*k02,c12=k01*k02-k00*k12,c22=k00*k11-k01*k01;
    const T det=k00*c00+k01*c01+k02*c02;
    const T inv=T(1)/det;
    const T a=(c00*L0+c01*L1+c02*L2)*inv;
    const T b=(c01*L0+c11*L1+c12*L2)*inv;
    const T c=(c02*L0+c12*L1+c22*L2)*inv;
    // dR = R W, W = [[0,-a,-b],[a,0,-c],[b,c,0]]
    T dR[9];
#pragma unroll
    for(int i=0;i<3;++i){
        const T r0=Re[3*i],r1=Re[3*i+1],r2=Re[3*i+2];
        dR[3*i]  = r1*a+r2*b;
        dR[3*i+1]=-r0*a+r2*c;
        dR[3*i+2]=-r0*b-r1*c;}
    T dH[9];cofactor3_diff(Fe,dF,dH);
    T HdF=T(0);
#pragma unroll
    for(int k=0;k<9;++k) HdF+=H[k]*dF[k];
    const T m2=T(2)*mu,lh=lambda*HdF,lj=lambda*(Je-T(1));
#pragma unroll
    for(int k=0;k<9;++k) dP[k]=m2*(dF[k]-dR[k])+lh*H[k]+lj*dH[k];
}

// The stress and the elastic Hessian of one particle in the rotation-free form of the
// transfers. With the left polar form F = S R (S symmetric), E = S - I, J = det F and dF = G F:
//   dF F^T = G S^2,  cof(F) F^T = J I,  cof(F):dF = J tr G,  d(cof F) F^T = J (tr G I - G^T),
// and R W R^T = W' solves W' S + S W' = M - M^T for M = G S, so that P of stress_P and dP of
// dP_dF become
//   V0 P F^T  = c1 E S + c3 I,
//   V0 dP F^T = c1 (M - W') S + c2 tr G I - c3 G^T,
//   c1 = 2 mu V0,  c3 = lambda V0 J (J - 1),  c2 = lambda V0 J^2 + c3.
// Nine numbers and about 110 operations per product instead of Fe, Re, lambda, mu and V0
// (21) and about 260. E is kept, not S, and formed from F - R, so that a small strain keeps
// its relative accuracy (the stress is as accurate as stress_P's from the same F and R). An
// EOS fluid has c1 = c3 = 0, its coefficient of the product in c2 and that of the explicit
// force in Exx.
template<class T> struct HessianData { T E[6],c1,c2,c3; };     // E: xx, xy, xz, yy, yz, zz
template<class T> MPM_HD void hessian_data(const T* F,const T* R,const T lambda,const T mu,const T Je,const T V0,HessianData<T>& h)
{
    T D[9],Q[9];
#pragma unroll
    for(int k=0;k<9;++k) D[k]=F[k]-R[k];
    mat_mul_bt(R,D,Q);
    h.E[0]=Q[0];h.E[1]=T(0.5)*(Q[1]+Q[3]);h.E[2]=T(0.5)*(Q[2]+Q[6]);
    h.E[3]=Q[4];h.E[4]=T(0.5)*(Q[5]+Q[7]);h.E[5]=Q[8];
    h.c1=T(2)*mu*V0;h.c3=lambda*V0*(Je*(Je-T(1)));h.c2=lambda*V0*(Je*Je)+h.c3;
}
// Inverse of the 3x3 matrix K of W' (entries 00, 01, 02, 11, 12, 22), S = I + E.
template<class T> MPM_HD void skew_system_inverse(const T* S,T* Ki)
{
    const T k00=S[3]+S[0],k01=S[4],k02=-S[2],k11=S[5]+S[0],k12=S[1],k22=S[5]+S[3];
    Ki[0]=k11*k22-k12*k12;Ki[1]=k02*k12-k01*k22;Ki[2]=k01*k12-k02*k11;
    Ki[3]=k00*k22-k02*k02;Ki[4]=k01*k02-k00*k12;Ki[5]=k00*k11-k01*k01;
    const T inv=T(1)/(k00*Ki[0]+k01*Ki[1]+k02*Ki[2]);
#pragma unroll
    for(int k=0;k<6;++k) Ki[k]*=inv;
}
// V0 P F^T (00, 01, 02, 11, 12, 22) of HessianData; an EOS fluid's pressure enters as -c I.
template<class T> MPM_HD void transfer_stress(const HessianData<T>& h,bool eos,T* A)
{
    const T* E=h.E;
    A[0]=h.c1*(E[0]+(E[0]*E[0]+E[1]*E[1]+E[2]*E[2]))+h.c3;
    A[1]=h.c1*(E[1]+(E[0]*E[1]+E[1]*E[3]+E[2]*E[4]));
    A[2]=h.c1*(E[2]+(E[0]*E[2]+E[1]*E[4]+E[2]*E[5]));
    A[3]=h.c1*(E[3]+(E[1]*E[1]+E[3]*E[3]+E[4]*E[4]))+h.c3;
    A[4]=h.c1*(E[4]+(E[1]*E[2]+E[3]*E[4]+E[4]*E[5]));
    A[5]=h.c1*(E[5]+(E[2]*E[2]+E[4]*E[4]+E[5]*E[5]))+h.c3;
    if(eos) A[0]=A[3]=A[5]=-E[0];
}

// A vector over the three components of a node value (FP64).
template<class T> struct C3 { T x,y,z; };
template<class T> MPM_HD C3<T> c3(T x,T y,T z){return C3<T>{x,y,z};}
MPM_HD C3<double> madd(const C3<double>& a,double s,const C3<double>& c){return C3<double>{fma(a.x,s,c.x),fma(a.y,s,c.y),fma(a.z,s,c.z)};}
MPM_HD C3<double> mul(const C3<double>& a,double s){return C3<double>{a.x*s,a.y*s,a.z*s};}
MPM_HD double cx(const C3<double>& a){return a.x;}
MPM_HD double cy(const C3<double>& a){return a.y;}

// B = V0 dP Fe^T from G, by columns (HessianData), and bg = B:G, the particle's part of
// s^T K s. FP32 solves the 3x3 system of the rotation part itself (hessian_stress2); FP64, whose
// arithmetic is 64 times slower against the same memory, reads the inverse that P2G stored.
template<class T> MPM_HD void hessian_stress(const C3<T> (&G)[3],const T* Sm,T c1,T c2,T cc3,const T* Ki,C3<T> (&B)[3],T& bg)
{
    const T S[3][3]={{Sm[0],Sm[1],Sm[2]},{Sm[1],Sm[3],Sm[4]},{Sm[2],Sm[4],Sm[5]}};
    C3<T> M[3];
#pragma unroll
    for(int j=0;j<3;++j) M[j]=madd(G[2],S[2][j],madd(G[1],S[1][j],mul(G[0],S[0][j])));
    const T L0=cy(M[0])-cx(M[1]),L1=M[0].z-cx(M[2]),L2=M[1].z-cy(M[2]);
    const T a=Ki[0]*L0+Ki[1]*L1+Ki[2]*L2,b=Ki[1]*L0+Ki[3]*L1+Ki[4]*L2,c=Ki[2]*L0+Ki[4]*L1+Ki[5]*L2;
    const C3<T> N[3]={c3<T>(cx(M[0]),cy(M[0])-a,M[0].z-b),c3<T>(cx(M[1])+a,cy(M[1]),M[1].z-c),c3<T>(cx(M[2])+b,cy(M[2])+c,M[2].z)};
    const T tr=c2*(cx(G[0])+cy(G[1])+G[2].z);
    // columns j of -c3 G^T (rows j of G), then c1 N S and the trace on the diagonal
    const C3<T> gt[3]={c3<T>(cx(G[0]),cx(G[1]),cx(G[2])),c3<T>(cy(G[0]),cy(G[1]),cy(G[2])),c3<T>(G[0].z,G[1].z,G[2].z)};
#pragma unroll
    for(int j=0;j<3;++j)
        B[j]=madd(N[2],c1*S[2][j],madd(N[1],c1*S[1][j],madd(N[0],c1*S[0][j],mul(gt[j],-cc3))));
    B[0]=c3<T>(cx(B[0])+tr,cy(B[0]),B[0].z);B[1]=c3<T>(cx(B[1]),cy(B[1])+tr,B[1].z);B[2]=c3<T>(cx(B[2]),cy(B[2]),B[2].z+tr);
    bg=T(0);
#pragma unroll
    for(int j=0;j<3;++j) bg+=cx(B[j])*cx(G[j])+cy(B[j])*cy(G[j])+B[j].z*G[j].z;
}

// The same of an EOS fluid, a trace: its E holds the pressure, of any size, and snow's 3x3
// system would take its third power (FP32 overflows above 1e13: 0 * inf in the force).
template<class T> MPM_HD void fluid_stress(const C3<T> (&G)[3],T c2,C3<T> (&B)[3],T& bg)
{
    const T g=cx(G[0])+cy(G[1])+G[2].z,tr=c2*g;
    B[0]=c3<T>(tr,T(0),T(0));B[1]=c3<T>(T(0),tr,T(0));B[2]=c3<T>(T(0),T(0),tr);
    bg=tr*g;
}

// Packed pairs of single-precision operations: one instruction does the work of two, and
// each half rounds exactly like the scalar fmaf / multiply / sum (their form in host code).
MPM_HD float2 pdup(float a){return make_float2(a,a);}
#if defined(__CUDA_ARCH__)&&__CUDA_ARCH__>=1000
MPM_HD float2 pfma(float2 a,float2 b,float2 c){return __ffma2_rn(a,b,c);}
MPM_HD float2 pmul(float2 a,float2 b){return __fmul2_rn(a,b);}
MPM_HD float2 padd(float2 a,float2 b){return __fadd2_rn(a,b);}
#else
MPM_HD float2 pfma(float2 a,float2 b,float2 c){return make_float2(fmaf(a.x,b.x,c.x),fmaf(a.y,b.y,c.y));}
MPM_HD float2 pmul(float2 a,float2 b){return make_float2(a.x*b.x,a.y*b.y);}
MPM_HD float2 padd(float2 a,float2 b){return make_float2(a.x+b.x,a.y+b.y);}
#endif
MPM_HD float2 psub(float2 a,float2 b){return pfma(b,make_float2(-1.f,-1.f),a);}   // exact product: rounds like a - b
// transfer_stress for two particles of snow.
MPM_HD void transfer_stress2(const float2 (&E)[6],float2 c1,float2 c3,float2 (&A)[6])
{
    auto dot=[&](int a,int b,int c,int d,int e,int f){return pfma(E[e],E[f],pfma(E[c],E[d],pmul(E[a],E[b])));};
    A[0]=pfma(c1,padd(E[0],dot(0,0,1,1,2,2)),c3);A[1]=pmul(c1,padd(E[1],dot(0,1,1,3,2,4)));
    A[2]=pmul(c1,padd(E[2],dot(0,2,1,4,2,5)));A[3]=pfma(c1,padd(E[3],dot(1,1,3,3,4,4)),c3);
    A[4]=pmul(c1,padd(E[4],dot(1,2,3,4,4,5)));A[5]=pfma(c1,padd(E[5],dot(2,2,4,4,5,5)),c3);
}
// B = V0 dP Fe^T from G for two particles (hessian_stress).
MPM_HD void hessian_stress2(const float2 (&G)[3][3],const float2 (&Sm)[6],float2 c1,float2 c2,float2 cc3,float2 (&B)[3][3],float2& bg)
{
    const int ix[3][3]={{0,1,2},{1,3,4},{2,4,5}};
    float2 M[3][3];
#pragma unroll
    for(int i=0;i<3;++i)
#pragma unroll
        for(int j=0;j<3;++j) M[i][j]=pfma(G[i][2],Sm[ix[2][j]],pfma(G[i][1],Sm[ix[1][j]],pmul(G[i][0],Sm[ix[0][j]])));
    // K a = L for the axial vector (a, b, c) of W' (skew_system_inverse)
    const float2 k00=padd(Sm[3],Sm[0]),k01=Sm[4],k02=pmul(Sm[2],pdup(-1.f)),k11=padd(Sm[5],Sm[0]),k12=Sm[1],k22=padd(Sm[5],Sm[3]);
    auto det2=[](float2 p,float2 q,float2 r,float2 s){return psub(pmul(p,q),pmul(r,s));};
    const float2 i00=det2(k11,k22,k12,k12),i01=det2(k02,k12,k01,k22),i02=det2(k01,k12,k02,k11);
    const float2 i11=det2(k00,k22,k02,k02),i12=det2(k01,k02,k00,k12),i22=det2(k00,k11,k01,k01);
    const float2 det=pfma(k02,i02,pfma(k01,i01,pmul(k00,i00)));
    const float2 inv=make_float2(1.f/det.x,1.f/det.y);
    const float2 L0=pmul(psub(M[1][0],M[0][1]),inv),L1=pmul(psub(M[2][0],M[0][2]),inv),L2=pmul(psub(M[2][1],M[1][2]),inv);
    const float2 a=pfma(i02,L2,pfma(i01,L1,pmul(i00,L0))),b=pfma(i12,L2,pfma(i11,L1,pmul(i01,L0))),c=pfma(i22,L2,pfma(i12,L1,pmul(i02,L0)));
    M[0][1]=padd(M[0][1],a);M[0][2]=padd(M[0][2],b);M[1][2]=padd(M[1][2],c);
    M[1][0]=psub(M[1][0],a);M[2][0]=psub(M[2][0],b);M[2][1]=psub(M[2][1],c);
    const float2 tr=pmul(c2,padd(padd(G[0][0],G[1][1]),G[2][2])),n3=pmul(cc3,pdup(-1.f));
    float2 cS[6];
#pragma unroll
    for(int k=0;k<6;++k) cS[k]=pmul(c1,Sm[k]);
#pragma unroll
    for(int i=0;i<3;++i)
#pragma unroll
        for(int j=0;j<3;++j){
            const float2 g=i==j?pfma(n3,G[j][i],tr):pmul(n3,G[j][i]);
            B[i][j]=pfma(M[i][2],cS[ix[2][j]],pfma(M[i][1],cS[ix[1][j]],pfma(M[i][0],cS[ix[0][j]],g)));
            bg=i==0&&j==0?pmul(B[i][j],G[i][j]):pfma(B[i][j],G[i][j],bg);}
}
MPM_HD void fluid_stress2(const float2 (&G)[3][3],float2 c2,float2 (&B)[3][3],float2& bg)
{
    const float2 g=padd(padd(G[0][0],G[1][1]),G[2][2]),tr=pmul(c2,g);
#pragma unroll
    for(int i=0;i<3;++i)
#pragma unroll
        for(int j=0;j<3;++j) B[i][j]=i==j?tr:pdup(0.f);
    bg=pmul(tr,g);
}

} // namespace mpm
